// Transmittance scan kernels: binning of developed crystals and the binned scan itself.
#include <type_traits>

#include "fg_internal.h"
#include "fg_pair.cuh"
#include "fg_scan.cuh"

namespace fg {

// Bin range [lo, hi] (um, padded by 1e-3) in one axis.
__device__ __forceinline__ void bin_span(double lo, double hi, float binw, uint32_t nb, uint32_t& b0, uint32_t& b1) {
  const float l = (static_cast<float>(lo) - 1e-3f) / binw, h = (static_cast<float>(hi) + 1e-3f) / binw;
  const float fl = fminf(fmaxf(floorf(l), 0.0f), (float)(nb - 1));
  const float fh = fminf(fmaxf(floorf(h), 0.0f), (float)(nb - 1));
  b0 = static_cast<uint32_t>(fl);
  b1 = static_cast<uint32_t>(fh);
}

// Bins of developed crystal s: those its leaf box overlaps (a ray outside the leaf box misses s).
__device__ __forceinline__ void leaf_bins(const ScanTile& t, uint32_t s, uint32_t& x0, uint32_t& x1, uint32_t& y0,
                                          uint32_t& y1) {
  const double* b = t.lbox64 + 6ull * t.leafof[s];
  bin_span(b[0], b[3], (float)(t.bin_px * t.pw), t.nbx, x0, x1);
  bin_span(b[1], b[4], (float)(t.bin_px * t.ph), t.nby, y0, y1);
}

__global__ void k_bin_count(ScanTile t, uint32_t* cnt) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= t.n || !t.developed[s]) return;
  uint32_t x0, x1, y0, y1;
  leaf_bins(t, s, x0, x1, y0, y1);
  for (uint32_t by = y0; by <= y1; ++by)
    for (uint32_t bx = x0; bx <= x1; ++bx) atomicAdd(&cnt[by * t.nbx + bx], 1u);
}

__global__ void k_bin_fill(ScanTile t, const uint32_t* off, uint32_t* cursor, uint32_t* items) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= t.n || !t.developed[s]) return;
  uint32_t x0, x1, y0, y1;
  leaf_bins(t, s, x0, x1, y0, y1);
  for (uint32_t by = y0; by <= y1; ++by)
    for (uint32_t bx = x0; bx <= x1; ++bx) {
      const uint32_t b = by * t.nbx + bx;
      items[off[b] + atomicAdd(&cursor[b], 1u)] = s;
    }
}

// Error-free transformations on floats (Knuth's two-sum, FMA two-product).
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
__device__ __forceinline__ void fast_two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  e = b - (s - a);
}
__device__ __forceinline__ void two_prod(float a, float b, float& p, float& e) {
  p = a * b;
  e = fmaf(a, b, -p);
}

// (ah + al) - (bh + bl) as a float pair, to about 2^-48 of the operands.
__device__ __forceinline__ void pair_sub(float ah, float al, float bh, float bl, float& h, float& l) {
  float s, e;
  two_sum(ah, -bh, s, e);
  two_sum(s, e + (al - bl), h, l);
}

// Fixed-point chord sums (units of 2^-40 um) without 64-bit integer / float conversions, which
// run on GB300's narrow FP64 pipe.  fix40(v) equals __float2ll_rn(v * 2^40) for 0 <= v < 2^15:
// below 2^31 the 32-bit conversion rounds the same way; above, v * 2^40 is an integer (its ulp is
// at least 2^8) split exactly into hi * 2^24 + lo.
__device__ __forceinline__ long long fix40(float v) {
  const float w = v * 1099511627776.0f;
  if (w < 2147483648.0f) return static_cast<long long>(__float2int_rn(w));
  const float hf = truncf(w * 0x1p-24f);
  const float lf = fmaf(-hf, 16777216.0f, w);  // exact: the low 24 bits of an integer
  return (static_cast<long long>(__float2int_rz(hf)) << 24) + __float2int_rz(lf);
}
// u rounded to the nearest float (ties to even), as __ll2float_rn does, in integer arithmetic.
__device__ __forceinline__ float u64_to_float_rn(unsigned long long u) {
  if (u < (1ull << 24)) return static_cast<float>(static_cast<uint32_t>(u));
  const int sh = 63 - __clzll(static_cast<long long>(u)) - 23;  // >= 1
  unsigned long long m = u >> sh;                                // 24 bits
  const unsigned long long rem = u & ((1ull << sh) - 1ull), half = 1ull << (sh - 1);
  if (rem > half || (rem == half && (m & 1ull))) ++m;            // m <= 2^24: exact as a float
  return static_cast<float>(static_cast<uint32_t>(m)) * __int_as_float((127 + sh) << 23);
}

// Crystal kinds in shared memory.
enum : int { K_CUBE = 0, K_CUBE_DF = 1, K_ELLIPSOID = 2, K_FP64 = 3 };

// Shared-memory image of a staged crystal (index c of the current chunk).  Coordinates are
// relative to the bin corner and carried as float pairs (hi + lo) so that ray-minus-crystal
// offsets are accurate to ~1e-8 um.  176 bytes, read as float4: 11 is odd, so the lanes of a warp,
// which test different crystals, spread over the banks.
struct __align__(16) Staged {
  float4 rect;        // x0, x1, y0, y1 (high words, with slack) outside of which no ray hits
  float4 c;           // centre: x hi, x lo, y hi, y lo
  float4 lbh, lbl;    // leaf box x0, x1, y0, y1: high words, low words
  float4 misc;        // delta, err, sig, kind (bits)
  float4 g[6];        // ScanPrep::g
};
struct ScanSmem {
  Staged k[SCAN_CH];
  int s[SCAN_CH];
  double T[SCAN_THREADS];
};

constexpr float EPS32 = 5.9604645e-8f;  // 2^-24

// Slack of a comparison on the high words of two coordinates of magnitude up to v (um): they differ
// from their float pairs by half an ulp each, and the difference rounds once more.
__device__ __forceinline__ float hi_slack(float v) { return 1e-4f + 5e-7f * v; }

// Stages crystal s for vertical rays relative to the bin corner (bx0, by0).  Everything is
// derived in FP64 once per crystal and CTA, then rounded:
//   cubes:      rows 0 and 1 of R as float pairs, 1 / (-R_2i), half-sizes as float pairs;
//   ellipsoids: R_0i / D_i, R_1i / D_i, e_i = -R_2i / D_i, A = |e|^2, 1 / A.
// Cubes whose faces are nearly parallel to the ray (|1/R_2i| > 15) evaluate their local origin in
// float-pair arithmetic; cubes with an exactly parallel face decide in FP64.
__device__ __forceinline__ void prep_crystal(const ScanTile& t, uint32_t s, ScanPrep& P) {
  const Crystal64 k = load64_parts(t, s);
  const double e64 = t.exp64[s];
  const double mdim = fmax(fmax(k.dims.x, k.dims.y), k.dims.z);
  const double m64 = __dmul_rn(mdim, e64);
  const float m = static_cast<float>(m64);
  split64(k.pos.x, P.ch[0], P.cl[0]);
  split64(k.pos.y, P.ch[1], P.cl[1]);
  const double* lb = t.lbox64 + 6ull * t.leafof[s];
  split64(lb[0], P.ch[2], P.cl[2]);
  split64(lb[3], P.ch[3], P.cl[3]);
  split64(lb[1], P.ch[4], P.cl[4]);
  split64(lb[4], P.ch[5], P.cl[5]);
  P.delta = static_cast<float>(t.z0 - k.pos.z);
  P.sig = t.sigma_c ? t.sigma_c[s] : t.sigma;
  const double x = k.q[0], y = k.q[1], z = k.q[2], w = k.q[3];
  // world = R local + p, so local_i = R_0i dx + R_1i dy + R_2i dz: rows 0..2 of R.
  const double R0[3] = {1.0 - 2.0 * (y * y + z * z), 2.0 * (x * y - z * w), 2.0 * (x * z + y * w)};
  const double R1[3] = {2.0 * (x * y + z * w), 1.0 - 2.0 * (x * x + z * z), 2.0 * (y * z - x * w)};
  const double R2[3] = {2.0 * (x * z - y * w), 2.0 * (y * z + x * w), 1.0 - 2.0 * (x * x + y * y)};
  const double D[3] = {k.dims.x * e64, k.dims.y * e64, k.dims.z * e64};
  float hx = 0.0f, hy = 0.0f;
  if (k.morph == 0) {
    float invmax = 0.0f;
    const float Dmax = static_cast<float>(fmax(fmax(D[0], D[1]), D[2]));
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      Pair r2;
      split64(-R2[i], r2.h, r2.l);
      const float inv = pair_quotf(1.0, -R2[i], Pair{1.0f, 0.0f}, r2);
      float r0, r0l, r1, r1l, d, dl;
      split64(R0[i], r0, r0l);
      split64(R1[i], r1, r1l);
      split64(D[i], d, dl);
      P.g[i] = make_float4(r0, r1, inv, d);
      P.g[3 + i] = make_float4(r0l, r1l, dl, 0.0f);
      invmax = fmaxf(invmax, fabsf(inv));
      hx += fabsf(r0 * d);  // a negative half-size acts by its magnitude
      hy += fabsf(r1 * d);
    }
    if (!(invmax < 1e30f)) {
      P.kind = K_FP64;
      P.err = INFINITY;
    } else if (invmax > 15.0f) {
      P.kind = K_CUBE_DF;
      P.err = 0.0f;  // bounds are formed per ray from the t values
    } else {
      P.kind = K_CUBE;
      // A cube lies within sqrt(3) m of its centre, so rays that can hit it are within mr of the
      // centre in x and y.  |d local| <= 4e-7 mr + 1e-7 (rounded rows, offsets); |d D| <= eps D;
      // each t = (+-D - lo) * inv carries (d lo + d D) |inv| + 2 eps |t|, with |t| <= (D + 2 mr)
      // invmax.
      const float mr = 1.7320509f * m;
      P.err = 4.0f * ((4e-7f * mr + 1e-7f + EPS32 * Dmax) * invmax + 2.0f * EPS32 * (Dmax + 2.0f * mr) * invmax);
    }
  } else {
    P.kind = K_ELLIPSOID;
    double A = 0.0;
    const double Dmin = fmin(fmin(D[0], D[1]), D[2]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double ei = -R2[i] / D[i];
      Pair r0, r1, d;
      split64(R0[i], r0.h, r0.l);
      split64(R1[i], r1.h, r1.l);
      split64(D[i], d.h, d.l);
      P.g[i] = make_float4(pair_quotf(R0[i], D[i], r0, d), pair_quotf(R1[i], D[i], r1, d), static_cast<float>(ei), 0.0f);
      P.g[3 + i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      A += ei * ei;
      const float u = r0.h * d.h, v = r1.h * d.h;
      hx += u * u;
      hy += v * v;
    }
    hx = sqrtf(hx);
    hy = sqrtf(hy);
    P.g[0].w = static_cast<float>(1.0 / A);
    // h = 1 - |P_perp|^2; P (|P| <= sqrt(2) m / Dmin) and P_perp = P + tc e carry ~8 eps |P|
    // each, so |d h| <= 2 |P_perp| 8 eps sqrt(3) Pmax + 4 eps; four times that as the bound.
    const float Pmax = static_cast<float>(1.4142135623730951 * m64 / Dmin);
    P.err = 4.0f * (2.0f * 1.05f * 8.0f * EPS32 * 1.7320508f * Pmax + 4.0f * EPS32) + 1e-9f;
  }
  P.g[4].w = hx * 1.0001f;
  P.g[5].w = hy * 1.0001f;
}

// Stages crystal s, whose bin-independent terms are P, for the bin whose 16-px-square corner is (bxh +
// bxl, byh + byl): those terms, and the centre and leaf box relative to the corner as float pairs
// (float arithmetic only).
__device__ __forceinline__ void stage_prepared(const ScanPrep& P, ScanSmem& sm, int c, uint32_t s, float bxh, float bxl,
                                               float byh, float byl) {
  Staged& S = sm.k[c];
  float4 ctr, lbh, lbl;
  pair_sub(P.ch[0], P.cl[0], bxh, bxl, ctr.x, ctr.y);
  pair_sub(P.ch[1], P.cl[1], byh, byl, ctr.z, ctr.w);
  pair_sub(P.ch[2], P.cl[2], bxh, bxl, lbh.x, lbl.x);
  pair_sub(P.ch[3], P.cl[3], bxh, bxl, lbh.y, lbl.y);
  pair_sub(P.ch[4], P.cl[4], byh, byl, lbh.z, lbl.z);
  pair_sub(P.ch[5], P.cl[5], byh, byl, lbh.w, lbl.w);
  // A hit lies within the geometry's extent and inside the leaf box.
  const float rx = P.g[4].w + hi_slack(fabsf(ctr.x)), ry = P.g[5].w + hi_slack(fabsf(ctr.z));
  S.rect = make_float4(fmaxf(ctr.x - rx, lbh.x - hi_slack(fabsf(lbh.x))), fminf(ctr.x + rx, lbh.y + hi_slack(fabsf(lbh.y))),
                       fmaxf(ctr.z - ry, lbh.z - hi_slack(fabsf(lbh.z))), fminf(ctr.z + ry, lbh.w + hi_slack(fabsf(lbh.w))));
  S.c = ctr;
  S.lbh = lbh;
  S.lbl = lbl;
  S.misc = make_float4(P.delta, P.err, P.sig, __int_as_float(P.kind));
#pragma unroll
  for (int i = 0; i < 6; ++i) S.g[i] = P.g[i];
  sm.s[c] = static_cast<int>(s);
}

// Out of line, for scans without prepared terms: inlined, the FP64 derivation would cost the scan's
// loops their registers.
static __device__ __noinline__ void stage_derived(const ScanTile& t, ScanSmem& sm, int c, uint32_t s, float bxh,
                                                  float bxl, float byh, float byl) {
  ScanPrep P;
  prep_crystal(t, s, P);
  stage_prepared(P, sm, c, s, bxh, bxl, byh, byl);
}

// stage_prepared with the terms from t.prep, or derived here.
__device__ __forceinline__ void stage_crystal(const ScanTile& t, ScanSmem& sm, int c, uint32_t s, float bxh,
                                              float bxl, float byh, float byl) {
  if (t.prep) {
    stage_prepared(t.prep[s], sm, c, s, bxh, bxl, byh, byl);
  } else {
    stage_derived(t, sm, c, s, bxh, bxl, byh, byl);
  }
}

// Staging terms of the listed developed crystals (their slots; *nlist of them, at most cap, or cap
// when nlist is null), once per crystal (k_scan reads them): one thread per listed crystal, so the
// FP64 derivation runs with every lane busy.
__global__ void k_scan_prep_list(const ScanTile* __restrict__ tiles, int ntiles, const uint32_t* __restrict__ list,
                                 const uint32_t* __restrict__ nlist, unsigned long long cap,
                                 ScanPrep* __restrict__ prep) {
  const unsigned long long i = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x;
  if (i >= cap || (nlist && i >= *nlist)) return;
  const unsigned long long g = list[i];
  int lo = 0, hi = ntiles - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tiles[mid].slot_base <= g) lo = mid; else hi = mid - 1;
  }
  const ScanTile& t = tiles[lo];
  const unsigned long long s = g - t.slot_base;
  if (s >= t.n || !t.developed[s]) return;
  ScanPrep P;
  prep_crystal(t, static_cast<uint32_t>(s), P);
  prep[g] = P;
}

void launch_scan_prep_list(const ScanTile* tiles, int ntiles, const uint32_t* list, const uint32_t* nlist,
                           unsigned long long cap, ScanPrep* prep, cudaStream_t st) {
  if (cap == 0) return;
  k_scan_prep_list<<<grid_for(cap, 128), 128, 0, st>>>(tiles, ntiles, list, nlist, cap, prep);
  FG_CUDA(cudaGetLastError());
}

// One thread's scanner ray in a bin: pixel, stratum and the ray origin relative to the corner of
// the 16-pixel square holding the bin (float pairs), shared by the forward scan and its adjoint.
struct ScanRay {
  uint32_t bin;
  bool active;
  float bxh, bxl, byh, byl;  // corner of the 16-pixel square holding the bin (um, float pairs)
  float oxh, oxl, oyh, oyl;
  float4 warp;     // x0, x1, y0, y1 of the warp's rays (high words)
};

// Pixel in the bin and stratum of thread tid.  A warp's pixels form a compact block (Morton order in
// bins of 2^k pixels: 4 x 2 pixels of 4 strata), so that it meets few crystals.
__device__ __forceinline__ void scan_place(const ScanTile& t, uint32_t tid, uint32_t& pix, uint32_t& lx, uint32_t& ly,
                                           uint32_t& st) {
  pix = tid / t.spp;
  st = tid % t.spp;
  const bool morton = (t.bin_px & (t.bin_px - 1)) == 0;
  lx = morton ? morton2_compact(pix) : pix % t.bin_px;
  ly = morton ? morton2_compact(pix >> 1) : pix / t.bin_px;
}

// The ray's place among the bin's: pixel-major in rows, strata in order.
__device__ __forceinline__ uint32_t scan_slot(const ScanTile& t, uint32_t tid) {
  uint32_t pix, lx, ly, st;
  scan_place(t, tid, pix, lx, ly, st);
  return pix < t.bin_px * t.bin_px ? (ly * t.bin_px + lx) * t.spp + st : SCAN_THREADS;
}

// The FP64 decision and chord of the calling thread's ray against crystal s (rare: the ray is formed
// anew here, so that the scan does not keep its pixel and stratum in registers).
static __device__ __noinline__ bool scan_chord_fp64(const ScanTile& t, uint32_t s, uint32_t bin, float& chord) {
  uint32_t pix, lx, ly, st;
  scan_place(t, threadIdx.x, pix, lx, ly, st);
  double ox, oy;
  scan_origin64(t, (bin % t.nbx) * t.bin_px + lx, (bin / t.nbx) * t.bin_px + ly, st % t.g, st / t.g, ox, oy);
  bool hit;
  chord = static_cast<float>(scan_chord64(t, s, ox, oy, hit));
  return hit;
}

// Decision and chord of one scanner ray against staged crystal c, whose rectangle holds the ray.  The
// ray's origin is a float pair relative to the bin's 16-px corner; a pair whose decision falls inside
// its error bound is decided with the reference's FP64 expressions (counted in nfb).
// DF: the crystal is a K_CUBE_DF (it is none otherwise).
template <bool DF>
__device__ __forceinline__ bool scan_pair(const ScanTile& t, const ScanSmem& sm, uint32_t c, const ScanRay& R, float& chord,
                                          uint32_t& nfb) {
  const float oxh = R.oxh, oxl = R.oxl, oyh = R.oyh, oyl = R.oyl;
  const Staged& S = sm.k[c];
  const float4 misc = S.misc, ctr = S.c, lb = S.lbh;
  const float delta = misc.x;
  const int kind = __float_as_int(misc.w);
  // Ray minus crystal centre, x and y, as float pairs.
  float dh, dl, dx, dxl, dy, dyl;
  two_sum(oxh, -ctr.x, dh, dl);
  fast_two_sum(dh, dl + (oxl - ctr.y), dx, dxl);
  two_sum(oyh, -ctr.z, dh, dl);
  fast_two_sum(dh, dl + (oyl - ctr.w), dy, dyl);
  // The leaf box (strict containment in x and y; the origin lies above every box in z): its margins
  // on the high words, and where those are too close to call, of float-pair differences, exact to
  // about 1e-12 um.
  float lm = fminf(fminf(oxh - lb.x, lb.y - oxh), fminf(oyh - lb.z, lb.w - oyh));
  if (fabsf(lm) <= hi_slack(fabsf(oxh) + fabsf(oyh))) {
    const float4 ll = S.lbl;
    float h, l;
    two_sum(oxh, -lb.x, h, l);
    lm = h + (l + (oxl - ll.x));
    two_sum(lb.y, -oxh, h, l);
    lm = fminf(lm, h + (l + (ll.y - oxl)));
    two_sum(oyh, -lb.z, h, l);
    lm = fminf(lm, h + (l + (oyl - ll.z)));
    two_sum(lb.w, -oyh, h, l);
    lm = fminf(lm, h + (l + (ll.w - oyl)));
  }
  const float EBL = 1e-9f;
  if (lm < -EBL) return false;
  bool amb = lm <= EBL || kind == K_FP64;
  bool hit = false;
  chord = 0.0f;
  if (!amb) {
    if (DF || kind != K_ELLIPSOID) {
      float tmin = -INFINITY, tmax = INFINITY;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const float4 gi = S.g[i];
        const float inv = gi.z, Dh = gi.w;
        float a1, a2;
        if (!DF) {
          const float lo_i = fmaf(gi.x, dx, gi.y * dy);
          a1 = -Dh - lo_i;
          a2 = Dh - lo_i;
        } else {
          // Local origin as a float pair, then the two face offsets exactly rounded.
          const float4 gl = S.g[3 + i];
          const float R0h = gi.x, R0l = gl.x, R1h = gi.y, R1l = gl.y, Dl = gl.z;
          float p0, e0, p1, e1, sh, sl;
          two_prod(R0h, dx, p0, e0);
          two_prod(R1h, dy, p1, e1);
          two_sum(p0, p1, sh, sl);
          sl += (e0 + e1) + ((R0h * dxl + R1h * dyl) + (R0l * dx + R1l * dy));
          float v, wv;
          two_sum(-Dh, -sh, v, wv);
          a1 = v + ((wv - Dl) - sl);
          two_sum(Dh, -sh, v, wv);
          a2 = v + ((wv + Dl) - sl);
        }
        const float t1 = a1 * inv, t2 = a2 * inv;
        tmin = fmaxf(tmin, fminf(t1, t2));
        tmax = fminf(tmax, fmaxf(t1, t2));
      }
      const float E = !DF ? misc.y : 4.0f * 3.0f * EPS32 * (fabsf(tmin) + fabsf(tmax)) + 1e-9f;
      const float m1 = tmax - tmin, m2 = tmax + delta;
      const float E2 = E + 4.0f * 3.0f * EPS32 * fabsf(delta) + 2e-6f;
      if (m1 > 2.0f * E && m2 > E2) {
        hit = true;
        chord = tmax - fmaxf(tmin, -delta);
      } else if (!(m1 < -2.0f * E || m2 < -E2)) {
        amb = true;
      }
    } else {
      float P[3];
      const float4 g0 = S.g[0], g1 = S.g[1], g2 = S.g[2];
      P[0] = fmaf(g0.x, dx, g0.y * dy);
      P[1] = fmaf(g1.x, dx, g1.y * dy);
      P[2] = fmaf(g2.x, dx, g2.y * dy);
      const float e0 = g0.z, e1 = g1.z, e2 = g2.z;
      const float iA = g0.w;
      // Closest approach along the ray (t' = tc) and the offset there: h = 1 - |P_perp|^2
      // has the sign of the reference's discriminant.
      const float tc = -(P[0] * e0 + P[1] * e1 + P[2] * e2) * iA;
      const float q0 = fmaf(tc, e0, P[0]), q1 = fmaf(tc, e1, P[1]), q2 = fmaf(tc, e2, P[2]);
      const float hh = 1.0f - (q0 * q0 + q1 * q1 + q2 * q2);
      const float E = misc.y;
      if (hh > E) {
        const float sq = sqrtf(hh * iA);
        const float t0 = tc - sq, t1 = tc + sq;
        const float E2 = 4.0f * 3.0f * EPS32 * (fabsf(t1) + fabsf(delta)) + 2e-6f;
        if (t1 + delta > E2) {
          hit = true;
          chord = t1 - fmaxf(t0, -delta);
        } else {
          amb = true;
        }
      } else if (!(hh < -E)) {
        amb = true;
      }
    }
  }
  if (amb) {
    ++nfb;
    hit = scan_chord_fp64(t, static_cast<uint32_t>(sm.s[c]), R.bin, chord);
  }
  return hit;
}

__device__ __forceinline__ ScanRay scan_ray(const ScanTile& t, uint32_t bin, uint32_t tid) {
  ScanRay R;
  R.bin = bin;
  const uint32_t bx = bin % t.nbx, by = bin / t.nbx;
  uint32_t pix, lx, ly, st;
  scan_place(t, tid, pix, lx, ly, st);
  const uint32_t px = bx * t.bin_px + lx, py = by * t.bin_px + ly;
  const bool active = pix < t.bin_px * t.bin_px && px < t.w && py < t.h;
  const uint32_t sx = st % t.g, sy = st / t.g;
  // Coordinates are taken relative to the corner of the 16-pixel square holding this bin, not to
  // the bin itself, so that every bin edge rounds identically and results do not depend on the
  // launch shape.
  const uint32_t ox_px = (bx * t.bin_px) & ~15u, oy_px = (by * t.bin_px) & ~15u;
  {
    // The corner as a whole number of jitter units, (ox_px g 2^24) (pw / (g 2^24)), in float pairs:
    // the ray offsets below are counted in the same units, so the two agree to about 2^-48.
    const float fx = static_cast<float>(ox_px * t.g) * 16777216.0f, fy = static_cast<float>(oy_px * t.g) * 16777216.0f;
    float p, e;
    two_prod(fx, t.jxh, p, e);
    fast_two_sum(p, fmaf(fx, t.jxl, e), R.bxh, R.bxl);
    two_prod(fy, t.jyh, p, e);
    fast_two_sum(p, fmaf(fy, t.jyl, e), R.byh, R.byl);
  }
  const uint32_t rlx = px - ox_px, rly = py - oy_px;  // < 16 + bin_px
  // Ray position relative to that corner as a float pair.  The offset in units of the 24-bit
  // jitter is an exact integer X = (l g + s) 2^24 + u, so x = X * pw / (g 2^24).
  float oxh = 0.0f, oxl = 0.0f, oyh = 0.0f, oyl = 0.0f;
  if (active) {
    const uint64_t ps = t.seed + static_cast<uint64_t>(px) * 0x9E3779B97F4A7C15ull +
                        static_cast<uint64_t>(py) * 0xC6A4A7935BD1E995ull;
    const P4 r = philox(sy * t.g + sx, 0, 0, TAG_SCAN, static_cast<uint32_t>(ps), static_cast<uint32_t>(ps >> 32));
    const float cxh = t.jxh, cxl = t.jxl, cyh = t.jyh, cyl = t.jyl;
    const uint32_t X = ((rlx * t.g + sx) << 24) + (r.x >> 8);
    const uint32_t Y = ((rly * t.g + sy) << 24) + (r.y >> 8);
    // X, Y < 2^31 as a float pair: Xh rounded, Xl = X - Xh exact (32-bit conversions only; the
    // 64-bit ones run on the FP64 pipe).
    const float Xh = __uint2float_rn(X), Yh = __uint2float_rn(Y);
    const float Xl = __int2float_rn(static_cast<int>(X - __float2uint_rn(Xh)));
    const float Yl = __int2float_rn(static_cast<int>(Y - __float2uint_rn(Yh)));
    float p, e;
    two_prod(Xh, cxh, p, e);
    fast_two_sum(p, e + (Xh * cxl + Xl * cxh), oxh, oxl);
    two_prod(Yh, cyh, p, e);
    fast_two_sum(p, e + (Yh * cyl + Yl * cyh), oyh, oyl);
  }
  R.active = active;
  R.oxh = oxh;
  R.oxl = oxl;
  R.oyh = oyh;
  R.oyl = oyl;
  float x0 = active ? oxh : INFINITY, x1 = active ? oxh : -INFINITY;
  float y0 = active ? oyh : INFINITY, y1 = active ? oyh : -INFINITY;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
    x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
    y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
    y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
  }
  R.warp = make_float4(x0, x1, y0, y1);
  return R;
}

// fn<DF>(c) for every staged crystal whose rectangle holds the ray.  The warp picks, 32 crystals at
// a time, those whose rectangle meets its rays, and each lane notes which of them hold its own ray;
// then every lane goes through its own crystals, so that a turn does not wait for the warp's other
// rays (they are hit by about a third of the same crystals).  The float-pair cubes (one in five of
// random orientation) are decided at once, all lanes together: their code is long, and the lanes'
// own turns would nearly always include one.  All 32 lanes call it.  (A NaN rejects nothing.)
template <class F>
__device__ __forceinline__ void scan_staged(const ScanSmem& sm, uint32_t cnt, const ScanRay& R, F&& fn) {
  static_assert(SCAN_CH == 128, "four words of candidates");
  const uint32_t lane = threadIdx.x & 31;
  uint32_t mine[4] = {0, 0, 0, 0};
#pragma unroll
  for (uint32_t w = 0; w < 4; ++w) {
    const uint32_t b = 32 * w;
    if (b >= cnt) break;
    bool near = b + lane < cnt, pair = false;
    if (near) {
      const Staged& S = sm.k[b + lane];
      const float4 r = S.rect;
      near = !(r.x > R.warp.y || r.y < R.warp.x || r.z > R.warp.w || r.w < R.warp.z);
      pair = __float_as_int(S.misc.w) == K_CUBE_DF;
    }
    const unsigned nm = __ballot_sync(0xffffffffu, near), pm = __ballot_sync(0xffffffffu, pair);
    for (unsigned m = nm & ~pm; m; m &= m - 1) {
      const float4 r = sm.k[b + __ffs(m) - 1].rect;
      if (!(R.oxh < r.x || R.oxh > r.y || R.oyh < r.z || R.oyh > r.w)) mine[w] |= m & (0u - m);
    }
    for (unsigned m = nm & pm; m; m &= m - 1) {
      const uint32_t c = b + __ffs(m) - 1;
      const float4 r = sm.k[c].rect;
      if (R.active && !(R.oxh < r.x || R.oxh > r.y || R.oyh < r.z || R.oyh > r.w)) fn(c, std::true_type{});
    }
  }
  if (!R.active) return;
  uint32_t b = 0;
  for (;;) {
    if (!mine[0]) {
      if (!(mine[1] | mine[2] | mine[3])) break;
      b += 32;
      mine[0] = mine[1];
      mine[1] = mine[2];
      mine[2] = mine[3];
      mine[3] = 0;
      continue;
    }
    const uint32_t c = b + __ffs(mine[0]) - 1;
    mine[0] &= mine[0] - 1;
    fn(c, std::false_type{});
  }
}

// Tile of global bin gb (last tile whose first bin <= gb).
__device__ __forceinline__ int scan_tile_of(const ScanTile* tiles, int ntiles, unsigned long long gb) {
  int lo = 0, hi = ntiles - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tiles[mid].bin_base <= gb) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// fn(pixel index, mean transmittance) for the bin's pixels, from the strata in sm.T.  Thread p
// finishes the bin's p-th pixel, so the FP64 work runs on consecutive lanes (a pixel's strata are spp
// consecutive entries; one thread in spp per pixel would leave most lanes of each FP64 instruction
// idle on GB300's narrow FP64 pipe).
template <class F>
__device__ __forceinline__ void scan_means(const ScanTile& t, const ScanSmem& sm, uint32_t bin, uint32_t tid, F&& fn) {
  const uint32_t a = t.spp;
  for (uint32_t p = tid; p * a < blockDim.x; p += blockDim.x) {
    const uint32_t bx = bin % t.nbx, by = bin / t.nbx;
    const uint32_t qx = bx * t.bin_px + p % t.bin_px, qy = by * t.bin_px + p / t.bin_px;
    if (p >= t.bin_px * t.bin_px || qx >= t.w || qy >= t.h) continue;
    // FP64 mean over strata in the reference's order (sy, sx), then f32 (transmittance.rs:142).
    double acc = 0.0;
    for (uint32_t k = 0; k < a; ++k) acc = __dadd_rn(acc, sm.T[p * a + k]);
    // Division by a power of two is the multiplication by its exact reciprocal.
    const float mean = (float)((a & (a - 1)) == 0 ? __dmul_rn(acc, 1.0 / static_cast<double>(a))
                                                   : __ddiv_rn(acc, static_cast<double>(a)));
    fn(static_cast<size_t>(qy) * t.w + qx, mean);
  }
}

// Adds a warp's FP64 decisions and hits to the counters (may be null).
__device__ __forceinline__ void scan_count(unsigned long long* stats, uint32_t nfb, uint32_t nh) {
  if (!stats) return;
  unsigned long long f = nfb, hsum = nh;
  for (int o = 16; o > 0; o >>= 1) {
    f += __shfl_down_sync(0xffffffffu, f, o);
    hsum += __shfl_down_sync(0xffffffffu, hsum, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (f) atomicAdd(&stats[1], f);
    if (hsum) atomicAdd(&stats[2], hsum);
  }
}

// What bounds it: issue slots (75 % issue activity at 21 of 32 lanes; DRAM 1 %).  A bin of 8 x 8
// tri-x pixels at full development stages 130 crystals; 30 of each 84 staged meet a warp's rays, and
// a ray is decided against 17 of them (scan_staged).  Testing every staged crystal for every ray,
// all lanes of a row of pixels in step, took 10.4 ms for a 2048 x 2048 px tri-x image (23.7 M rays,
// 390 M hits); culling by warp 6.0; the lanes' own lists, with the float-pair cubes decided
// together, 5.3.
//
// Launch bounds of 4 x 256 threads per SM (64 registers; 3: 9.5 against 8.9 ms for the scan stage):
// more CTAs in flight cover the staging and the FP64 fallbacks.
__global__ void __launch_bounds__(SCAN_THREADS, 4) k_scan(const ScanTile* __restrict__ tiles,
                                                       int ntiles, uint32_t* err,
                                                       unsigned long long* stats) {
  __shared__ ScanSmem sm;
  const unsigned long long gb = blockIdx.x;
  const ScanTile& t = tiles[scan_tile_of(tiles, ntiles, gb)];
  const uint32_t bin = static_cast<uint32_t>(gb - t.bin_base);
  const uint32_t a = t.spp;
  const uint32_t tid = threadIdx.x;
  const ScanRay R = scan_ray(t, bin, tid);
  const bool active = R.active;
  long long Lfix = 0;  // chord sum (sigma-weighted when per crystal), 2^-40 um units
  uint32_t nh = 0, nfb = 0;
  const uint32_t b0 = min(t.bin_off[bin], t.items_cap), b1 = min(t.bin_off[bin + 1], t.items_cap);
  const bool per_crystal = t.sigma_c != nullptr;
  for (uint32_t base = b0; base < b1; base += SCAN_CH) {
    const uint32_t cnt = min(static_cast<uint32_t>(SCAN_CH), b1 - base);
    __syncthreads();
    for (uint32_t c = tid; c < cnt; c += blockDim.x)
      stage_crystal(t, sm, c, t.bin_items[base + c], R.bxh, R.bxl, R.byh, R.byl);
    __syncthreads();
    scan_staged(sm, cnt, R, [&](uint32_t c, auto df) {
      float chord;
      if (!scan_pair<decltype(df)::value>(t, sm, c, R, chord, nfb)) return;
      ++nh;
      const float v = per_crystal ? sm.k[c].misc.z * fmaxf(chord, 0.0f) : fmaxf(chord, 0.0f);
      Lfix += fix40(v);
    });
  }
  float T = 1.0f;
  if (active) {
    // Lfix * 2^-40 rounded once to float (the conversion rounds, the power-of-two scale is exact).
    const float L = u64_to_float_rn(static_cast<unsigned long long>(Lfix)) * 0x1p-40f;
    T = per_crystal ? expf(-L) : expf(-t.sigma * L);
    if (t.ray_hits) {
      uint32_t pix, lx, ly, st;
      scan_place(t, tid, pix, lx, ly, st);
      const uint32_t px = (bin % t.nbx) * t.bin_px + lx, py = (bin / t.nbx) * t.bin_px + ly;
      t.ray_hits[(static_cast<size_t>(py) * t.w + px) * a + st] = static_cast<uint16_t>(min(nh, 65535u));
    }
  }
  const uint32_t slot = scan_slot(t, tid);
  if (slot < SCAN_THREADS) sm.T[slot] = f2d_exact(T);
  __syncthreads();
  scan_means(t, sm, bin, tid, [&](size_t idx, float mean) {
    float v;
    if (t.mode == 0) {
      v = mean;
    } else if (t.mode == 1) {
      v = 1.0f - mean;
    } else {
      const float tt = fmaxf(mean, 1e-4f);
      v = fminf(fmaxf(-log10f(tt) / 3.0f, 0.0f), 1.0f);
    }
    if (t.out) t.out[idx] = v;
    if (t.image8) t.image8[idx] = static_cast<uint8_t>(rintf(fminf(fmaxf(v, 0.0f), 1.0f) * 255.0f));
    // The mean transmittance; launch_density turns it into the density in a pass of its own.
    if (t.d_neg) t.d_neg[idx] = mean;
  });
  scan_count(stats, nfb, nh);
}

// Adjoint of k_scan with respect to the per-crystal opacities (single tile).  The forward is
// recomputed from the developed mask: pass 1 forms each ray's optical depth exactly as k_scan
// does and writes the pixels' transmittance; pass 2 stages the bin's crystals again (unless all of
// them are still there) and adds w[p] / spp * T_ray * chord_s for every hit to a per-crystal FP64 sum
// in shared memory, flushed with one global atomic per staged crystal.
//
// Bound by issue, as k_scan.  Four CTAs per SM (64 registers) as there: a gradient step takes 4.39 ms with the two
// that 126 registers leave, 4.16 with three, 4.04 with four (spills included).
__global__ void __launch_bounds__(SCAN_THREADS, 4) k_scan_adjoint(const ScanTile* __restrict__ tiles,
                                                               const float* __restrict__ wpx,
                                                               double* __restrict__ g, float* __restrict__ Tpx,
                                                               unsigned long long* stats) {
  __shared__ ScanSmem sm;
  __shared__ double gsum[SCAN_CH];
  const ScanTile& t = tiles[0];
  const uint32_t bin = blockIdx.x;
  const uint32_t a = t.spp;
  const uint32_t tid = threadIdx.x;
  const ScanRay R = scan_ray(t, bin, tid);
  const uint32_t b0 = min(t.bin_off[bin], t.items_cap), b1 = min(t.bin_off[bin + 1], t.items_cap);
  const bool per_crystal = t.sigma_c != nullptr;
  uint32_t nfb = 0, nh = 0;
  long long Lfix = 0;
  for (uint32_t base = b0; base < b1; base += SCAN_CH) {
    const uint32_t cnt = min(static_cast<uint32_t>(SCAN_CH), b1 - base);
    __syncthreads();
    for (uint32_t c = tid; c < cnt; c += blockDim.x)
      stage_crystal(t, sm, c, t.bin_items[base + c], R.bxh, R.bxl, R.byh, R.byl);
    __syncthreads();
    scan_staged(sm, cnt, R, [&](uint32_t c, auto df) {
      float chord;
      if (!scan_pair<decltype(df)::value>(t, sm, c, R, chord, nfb)) return;
      ++nh;
      const float v = per_crystal ? sm.k[c].misc.z * fmaxf(chord, 0.0f) : fmaxf(chord, 0.0f);
      Lfix += fix40(v);
    });
  }
  scan_count(stats, nfb, nh);  // the forward's
  float coef = 0.0f, T = 1.0f;
  if (R.active) {
    const float L = u64_to_float_rn(static_cast<unsigned long long>(Lfix)) * 0x1p-40f;  // as in k_scan
    T = per_crystal ? expf(-L) : expf(-t.sigma * L);
    uint32_t pix, lx, ly, st;
    scan_place(t, tid, pix, lx, ly, st);
    const uint32_t px = (bin % t.nbx) * t.bin_px + lx, py = (bin / t.nbx) * t.bin_px + ly;
    coef = wpx[static_cast<size_t>(py) * t.w + px] / static_cast<float>(a) * T;
  }
  const uint32_t slot = scan_slot(t, tid);
  if (slot < SCAN_THREADS) sm.T[slot] = f2d_exact(T);
  __syncthreads();
  scan_means(t, sm, bin, tid, [&](size_t idx, float mean) { Tpx[idx] = mean; });
  for (uint32_t base = b0; base < b1; base += SCAN_CH) {
    const uint32_t cnt = min(static_cast<uint32_t>(SCAN_CH), b1 - base);
    __syncthreads();
    for (uint32_t c = tid; c < cnt; c += blockDim.x) {
      if (b1 - b0 > SCAN_CH) stage_crystal(t, sm, c, t.bin_items[base + c], R.bxh, R.bxl, R.byh, R.byl);
      gsum[c] = 0.0;
    }
    __syncthreads();
    scan_staged(sm, cnt, R, [&](uint32_t c, auto df) {
      if (coef == 0.0f) return;
      float chord;
      if (scan_pair<decltype(df)::value>(t, sm, c, R, chord, nfb))
        atomicAdd(&gsum[c], static_cast<double>(coef) * static_cast<double>(fmaxf(chord, 0.0f)));
    });
    __syncthreads();
    for (uint32_t c = tid; c < cnt; c += blockDim.x)
      if (gsum[c] != 0.0) atomicAdd(&g[sm.s[c]], gsum[c]);
  }
}

// d = -log10(clamp(T, 1e-4, 1)) + 0.05 as FP64 rounded to float (image_pipeline.rs:1007-1011), in
// place over the pixels' mean transmittance; evaluated as a pair of floats, FP64 where that does not
// settle the rounding (4.2 M px: 400 us in FP64 alone).
// A pass of its own so that every lane of a warp converts a pixel: inside k_scan only one thread per
// pixel (of spp) would.
__global__ void k_density(float* __restrict__ d, unsigned long long n) {
  const unsigned long long stride = static_cast<unsigned long long>(gridDim.x) * blockDim.x;
  for (unsigned long long i = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; i < n;
       i += stride)
    d[i] = pair_densityf(d[i]);
}

void launch_density(float* d, unsigned long long n, cudaStream_t st) {
  if (n == 0) return;
  k_density<<<static_cast<unsigned>(std::min<unsigned long long>(grid_for(n, 256), 152ull * 16)), 256, 0, st>>>(d, n);
  FG_CUDA(cudaGetLastError());
}

void launch_scan(const ScanTile* tiles, int ntiles, unsigned long long nbins, unsigned threads, uint32_t* err,
                 unsigned long long* stats, cudaStream_t st) {
  if (nbins == 0) return;
  k_scan<<<static_cast<unsigned>(nbins), threads, 0, st>>>(tiles, ntiles, err, stats);
  FG_CUDA(cudaGetLastError());
}

// Chooses the bin edge so one CTA holds bin_px^2 pixels of `spp` strata.
uint32_t scan_bin_px(uint32_t spp) {
  uint32_t b = 1;
  while ((b + 1) * (b + 1) * spp <= SCAN_THREADS) ++b;
  return b;
}

// Bins the developed crystals of an emulsion for a scan: descriptor, bin offsets and lists on the
// device (shared by the forward scan and its adjoint).
struct ScanPlan {
  ScanTile t{};
  RTreeBufs tree;             // the reference tree over the developed crystals
  DBuf<uint32_t> tree_list;
  DBuf<ScanPrep> prep;
  DBuf<uint32_t> cnt, off, cur, items;
  DBuf<ScanTile> td;
  unsigned nbins = 0, threads = 0;
};

uint32_t scan_grid(const fg_scan_cfg& cfg) {
  const uint32_t spp_req = std::max<uint32_t>(cfg.samples_per_pixel, 1);
  const uint32_t g = static_cast<uint32_t>(std::lround(std::sqrt(static_cast<double>(spp_req))));
  FG_REQUIRE(std::max<uint32_t>(g * g, 1) <= SCAN_THREADS, "samples_per_pixel too large (at most 256 strata)");
  FG_REQUIRE(cfg.width_px > 0 && cfg.height_px > 0, "scan size must be positive");
  return g;
}

static void plan_scan(fg_engine* e, const fg_emulsion* em, const fg_scan_cfg& cfg, uint64_t seed,
                      const float* sigma_sorted, const ScanOut& out, ScanPlan& P) {
  cudaStream_t st = e->stream;
  const uint32_t g = scan_grid(cfg), a = std::max<uint32_t>(g * g, 1);
  build_emulsion_tree(e, em, true, P.tree, P.tree_list, false);
  ScanTile& t = P.t;
  t = ScanTile{};
  t.lbox64 = P.tree.box64.p;
  t.leafof = P.tree.leafof.p;
  t.a = em->a.p;
  t.q = em->q.p;
  t.d = em->d.p;
  t.pos64 = em->has64 ? em->pos64.p : nullptr;
  t.dims64 = em->has64 ? em->dims64.p : nullptr;
  t.quat64 = em->has64 ? em->quat64.p : nullptr;
  t.developed = em->developed.p;
  t.exp64 = em->exp64.p;
  t.sigma_c = sigma_sorted;
  t.out = out.out;
  t.image8 = out.image8;
  t.d_neg = out.d_neg;
  t.ray_hits = out.ray_hits;
  t.pw = em->cfg.width / static_cast<double>(cfg.width_px);
  t.ph = em->cfg.height / static_cast<double>(cfg.height_px);
  t.z0 = em->cfg.depth + 0.1;
  t.seed = seed;
  t.bin_base = 0;
  t.w = cfg.width_px;
  t.h = cfg.height_px;
  t.g = g;
  t.spp = a;
  t.bin_px = scan_bin_px(a);
  t.nbx = (t.w + t.bin_px - 1) / t.bin_px;
  t.nby = (t.h + t.bin_px - 1) / t.bin_px;
  t.n = em->n;
  t.sigma = static_cast<float>(cfg.silver_opacity);
  t.mode = cfg.mode;
  set_jitter_units(t);
  const size_t nbins = static_cast<size_t>(t.nbx) * t.nby;
  FG_REQUIRE(nbins < 0x80000000ull, "scan too large");
  P.nbins = static_cast<unsigned>(nbins);
  P.cnt.alloc(nbins + 1, st);
  P.off.alloc(nbins + 1, st);
  P.cur.alloc(nbins, st);
  FG_CUDA(cudaMemsetAsync(P.cnt.p, 0, (nbins + 1) * sizeof(uint32_t), st));
  FG_CUDA(cudaMemsetAsync(P.cur.p, 0, nbins * sizeof(uint32_t), st));
  if (em->n) k_bin_count<<<grid_for(em->n, 256), 256, 0, st>>>(t, P.cnt.p);
  exclusive_scan_u32(P.cnt.p, P.off.p, nbins + 1, st);
  uint32_t total = 0;
  FG_CUDA(cudaMemcpyAsync(&total, P.off.p + nbins, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  FG_CUDA(cudaStreamSynchronize(st));
  P.items.alloc(std::max<uint32_t>(total, 1), st);
  if (em->n) k_bin_fill<<<grid_for(em->n, 256), 256, 0, st>>>(t, P.off.p, P.cur.p, P.items.p);
  t.bin_off = P.off.p;
  t.bin_items = P.items.p;
  t.items_cap = total;
  t.slot_base = 0;
  P.prep.alloc(std::max<uint32_t>(em->n, 1), st);
  t.prep = P.prep.p;
  P.td.alloc(1, st);
  FG_CUDA(cudaMemcpyAsync(P.td.p, &t, sizeof(ScanTile), cudaMemcpyHostToDevice, st));
  launch_scan_prep_list(P.td.p, 1, P.tree_list.p, nullptr, P.tree.count, P.prep.p, st);
  // Whole warps only: the closing reductions shuffle across all 32 lanes.
  P.threads = ((t.bin_px * t.bin_px * a + 31) / 32) * 32;
}

void scan(fg_engine* e, const fg_emulsion* em, const fg_scan_cfg& cfg, uint64_t seed,
          const float* sigma_sorted, const ScanOut& out) {
  ScanPlan P;
  plan_scan(e, em, cfg, seed, sigma_sorted, out, P);
  k_scan<<<P.nbins, P.threads, 0, e->stream>>>(P.td.p, 1, e->d_err, e->d_stats);
  FG_CUDA(cudaGetLastError());
  if (out.d_neg) launch_density(out.d_neg, static_cast<unsigned long long>(cfg.width_px) * cfg.height_px, e->stream);
  FG_CUDA(cudaStreamSynchronize(e->stream));
}

// Adjoint of the scan with respect to the per-crystal opacities: g[s] += sum over the rays of
// pixel p of w[p] / spp * T_ray * chord_s (w = dL/dT of the pixel, T_ray the ray's transmittance).
void scan_adjoint(fg_engine* e, const fg_emulsion* em, const fg_scan_cfg& cfg, uint64_t seed,
                  const float* sigma_sorted, const float* wpx, double* g_sorted, float* T) {
  ScanPlan P;
  plan_scan(e, em, cfg, seed, sigma_sorted, ScanOut{}, P);
  k_scan_adjoint<<<P.nbins, P.threads, 0, e->stream>>>(P.td.p, wpx, g_sorted, T, e->d_stats);
  FG_CUDA(cudaGetLastError());
  FG_CUDA(cudaStreamSynchronize(e->stream));
}

}  // namespace fg
