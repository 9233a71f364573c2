// Host-side internals shared by the translation units of libfgrain_cuda.so.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/fgrain_cuda.h"
#include "fg_cells.cuh"
#include "fg_device.cuh"
#include "fg_rtree.cuh"
#include "fg_transport.cuh"

namespace fg {

// A failed CUDA call or a rejected argument, carried to the C boundary as (status, message).
struct Error {
  fg_status st;
  std::string msg;
};

#define FG_CUDA(call)                                                                     \
  do {                                                                                    \
    cudaError_t e__ = (call);                                                             \
    if (e__ != cudaSuccess) throw ::fg::Error{::fg::status_of(e__), std::string(#call) + \
                                              ": " + cudaGetErrorString(e__)};            \
  } while (0)

#define FG_REQUIRE(cond, msg)                                                   \
  do {                                                                          \
    if (!(cond)) throw ::fg::Error{FG_ERR_INVALID_ARG, std::string(msg)};       \
  } while (0)

inline fg_status status_of(cudaError_t e) {
  switch (e) {
    case cudaErrorMemoryAllocation: return FG_ERR_OOM;
    case cudaErrorInvalidDevice:
    case cudaErrorNoDevice:
    case cudaErrorInsufficientDriver: return FG_ERR_ADAPTER_NOT_FOUND;
    case cudaErrorInvalidValue: return FG_ERR_INVALID_ARG;
    default: return FG_ERR_PIPELINE;
  }
}

// Device bytes held through DBuf and the optional cap on them (fg_set_device_budget).
inline std::atomic<unsigned long long> g_dev_bytes{0};
inline std::atomic<unsigned long long> g_dev_budget{0};

// Device buffer owned by RAII; stream-ordered allocation on the engine stream.  view() makes it a
// non-owning window onto memory that someone else holds (nothing is freed then).
template <class T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  cudaStream_t s = nullptr;
  bool own = true;
  DBuf() = default;
  DBuf(size_t count, cudaStream_t st) { alloc(count, st); }
  void alloc(size_t count, cudaStream_t st) {
    release();
    s = st;
    own = true;
    if (!count) return;
    const unsigned long long bytes = count * sizeof(T), cap = g_dev_budget.load();
    if (cap && g_dev_bytes.fetch_add(bytes) + bytes > cap) {
      g_dev_bytes.fetch_sub(bytes);
      throw Error{FG_ERR_OOM, "device budget of " + std::to_string(cap) + " bytes exceeded (fg_set_device_budget)"};
    }
    if (!cap) g_dev_bytes.fetch_add(bytes);
    const cudaError_t r = cudaMallocAsync(reinterpret_cast<void**>(&p), bytes, st);
    if (r != cudaSuccess) {
      g_dev_bytes.fetch_sub(bytes);
      p = nullptr;
      throw Error{status_of(r), std::string("cudaMallocAsync: ") + cudaGetErrorString(r)};
    }
    n = count;
  }
  void view(T* ptr, size_t count) {
    release();
    p = ptr;
    n = count;
    own = false;
  }
  void release() {
    if (p && own) {
      cudaFreeAsync(p, s);
      g_dev_bytes.fetch_sub(n * sizeof(T));
    }
    p = nullptr;
    n = 0;
    own = true;
  }
  ~DBuf() { release(); }
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  DBuf(DBuf&& o) noexcept : p(o.p), n(o.n), s(o.s), own(o.own) { o.p = nullptr; o.n = 0; }
  DBuf& operator=(DBuf&& o) noexcept {
    if (this != &o) { release(); p = o.p; n = o.n; s = o.s; own = o.own; o.p = nullptr; o.n = 0; }
    return *this;
  }
};

// Stage timer: events recorded on the engine stream around each stage.
struct StageTimer {
  cudaEvent_t ev[2 * 8];
  int used = 0;
  bool made = false;
  void init() {
    if (made) return;
    for (auto& e : ev) FG_CUDA(cudaEventCreate(&e));
    made = true;
  }
  void destroy() {
    if (!made) return;
    for (auto& e : ev) cudaEventDestroy(e);
    made = false;
  }
};

// fg_rtree.cu: device buffers of reference-tree builds over the tiles of a batch (or one
// emulsion).  Element positions and nodes are laid out tile after tile (RTile::ebase, nbase).
struct RTreeBufs {
  int ntiles = 0;
  int levels = 0;                 // most global split levels before the per-block finish
  int wpw = 8;                    // words per warp of the levels' chunks
  unsigned long long E = 0, N = 0, nblk = 0;
  uint32_t count = 0;             // elements of a one-tile tree built on the host's request
  DBuf<RTile> tiles;
  DBuf<uint32_t> idx0, idx1, nof0, nof1, bits, wp, P, Q;
  DBuf<unsigned long long> blk;         // running sum of the big flags, per chunk of positions
  DBuf<unsigned long long> key0, key1;  // three ordered centroid keys per element (SoA), travelling with the order
  DBuf<uint32_t> ridx;            // final element order (slots): a leaf's crystals in reference order
  DBuf<unsigned long long> acc;   // per node: ordered centroid minima, maxima (3 each)
  DBuf<double> box64;             // per node: lo xyz, hi xyz (FP64, exact)
  DBuf<uint32_t> parent;          // per node: parent id (0xffffffff for a root)
  DBuf<uint32_t> nstart, ncount, ntile, ndepth;
  DBuf<int> nsplit;               // split axis, -1 for a leaf
  DBuf<int2> nchild;              // global ids of the children
  DBuf<unsigned long long> nthr;  // split threshold (a key)
  DBuf<uint32_t> wl0, wl1, bq, bqpar, cnt;  // worklists (wl0 then the refit's arrival counts), block
                                            // queue (node, buffer parity), counts and chunk starts
  unsigned long long R = 0;       // walk records (all tiles)
  DBuf<Node4> rnode;              // four-wide walk records (tile-local refs)
  DBuf<uint2> rleaf;              // leaf: first element (tile-local position), count
  DBuf<uint32_t> leafof;          // optional: leaf id of each element slot
  DBuf<uint32_t> rank;            // optional: place of each element slot in the reference walk's order
};

// An emulsion's cells as they are built: the descriptor, and what is found of the set.
struct CellFit {
  TileDesc tile;
  double uneven;   // launch_cells_uneven
  uint32_t unfit;  // k_cells_count
};

// fg_cells.cu: the crystals of a batch's tiles (or one emulsion) in cells (CellGrid).
struct CellBufs {
  unsigned long long ncells = 0;
  DBuf<uint32_t> cnt, off, place;  // per cell: crystals, first position; per slot: its position
  DBuf<float4> pos, q, d, leaf;
  DBuf<uint2> by_rank;
  void alloc(unsigned long long ncap, unsigned long long cells, cudaStream_t st);
  // Sets the pointers of one tile's grid (cell_base set, first crystal slot cbase).
  void attach(CellGrid& g, unsigned long long cbase) const;
};
}  // namespace fg

struct fg_engine {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::recursive_mutex mu;
  std::string err;
  std::string name;
  uint32_t* d_err = nullptr;                    // device error word
  unsigned long long* d_stats = nullptr;        // device counters (hits, fallbacks, ...)
  fg_timings timings{};
  int sm_count = 0;
  fg::StageTimer timer;
};

struct fg_emulsion {
  fg_emulsion_cfg cfg{};
  uint32_t n = 0;
  cudaStream_t stream = nullptr;
  // Hot crystal records in Morton order.
  fg::DBuf<float4> a, q, d;
  // FP64 copies (uploaded sets only).
  fg::DBuf<double> pos64, dims64, quat64, sens64;
  fg::DBuf<uint32_t> sorted_to_id, id_to_sorted;
  // The reference tree over all crystals in id order (the transport walks, the development's
  // radius queries).
  fg::RTreeBufs rt;
  // The crystals in cells for the transport and the touch queries; grid.x.n is 0 for sets that stay
  // on the tree walk (build_emulsion_cells).
  fg::CellBufs cells;
  fg::CellGrid grid{};
  fg::DBuf<fg::CellFit> fit;        // its descriptor in device memory (device code reads the axes as vectors)
  // Mutable per-crystal state (Morton order).
  fg::DBuf<uint32_t> counts;
  fg::DBuf<uint8_t> developed;
  fg::DBuf<float> exp32;
  fg::DBuf<double> exp64;
  fg::DBuf<int64_t> clump;  // by crystal id
  bool has64 = false;
  double extent = 0.0;             // largest coordinate magnitude (sets the box padding)
  double max_half_dim = 0.0;       // largest crystal half-dimension (sets the walks' reach)
  double mean_area = 0.0;          // mean projected area of a crystal, um^2 (cells_area)
  bool any_cubic = true;           // some crystal is a cube (only a cube reaches out of its box)
  std::vector<uint32_t> h_s2id;    // host copy of sorted_to_id (empty: identity)

  fg::CrystalsView view() const {
    fg::CrystalsView v;
    v.a = a.p; v.q = q.p; v.d = d.p;
    v.pos64 = has64 ? pos64.p : nullptr;
    v.dims64 = has64 ? dims64.p : nullptr;
    v.quat64 = has64 ? quat64.p : nullptr;
    v.sens64 = has64 ? sens64.p : nullptr;
    v.n = n;
    return v;
  }
};

namespace fg {

// fg_bvh.cu
// Sorts crystals by Morton code and fills the hot arrays; returns the sorted keys.
// pos_host / pos_dev: id-ordered FP64 positions on the host and on the device.
void morton_order(fg_emulsion* em, const double* pos_host, const double* pos_dev, cudaStream_t st,
                  DBuf<uint64_t>& keys, DBuf<uint32_t>& order);
void gather_sorted(fg_emulsion* em, const uint32_t* order, const double* pos, const double* dims,
                   const double* quat, const double* sens, const int32_t* morph, int32_t morph_all,
                   cudaStream_t st);

// fg_cells.cu, fg_transport.cu: the emulsion's cells, when they suit its crystals (after its tree).
void build_emulsion_cells(fg_engine* e, fg_emulsion* em);

// Sets RTile::ebase / nbase / ncap from ecap, copies the tiles to the device and allocates.  The
// caller fills the source pointers and ecap of each tile, and RTile::n (and order) on the device
// before each build.
// Each tile gets min(ecap + 2, node_frac * ecap + 64) nodes (the reference tree has about 0.67
// nodes per element; running out fails the build with the list-overflow error bit).
// leafof (when wanted) gets max(elements, leafof_slots) words: it is indexed by element slot.
// rank (when wanted) gets as many.
void rtree_alloc(RTreeBufs& B, std::vector<RTile>& tiles, bool want_leafof, cudaStream_t st, double node_frac = 1.0,
                 size_t leafof_slots = 0, bool want_rank = false, bool walks = true);
// Enqueues a build (capturable: no host synchronisation).  tiles_dev (optional) replaces the tile
// array of the allocation by one with the same layout (ebase, nbase, ecap, ncap) but other element
// sources, so that one set of buffers serves several trees in turn.
// walks: also the boxes above the leaves and the walk records (a build that only gives leaves, ranks
// and leaf boxes does without).  key32: every tile's crystals are finite FP32 records without FP64
// copies and without expansion (then their centroids are their positions).
void rtree_build(RTreeBufs& B, uint32_t* err, cudaStream_t st, bool walks, bool key32, RTile* tiles_dev = nullptr);
unsigned rtree_kernel_launches(const RTreeBufs& B, bool walks);
// One tile's build in memory the caller holds (nothing allocated): bytes needed for a tile of ecap
// elements, and the attach that carves every buffer (the tile descriptor too) from `base`
// (256-byte aligned).  The tile's source pointers are set by the caller; tile.n may be written on
// the device later (RTreeBufs::tiles.p).
size_t rtree_scratch_bytes(uint32_t ecap, bool want_leafof, uint32_t leafof_slots);
void rtree_attach(RTreeBufs& B, RTile tile, bool want_leafof, uint32_t leafof_slots, unsigned char* base,
                  size_t bytes, cudaStream_t st);
// The tree of an emulsion over all its crystals, or over its developed crystals with their
// expansion (the scan's tree, transmittance.rs:86-89), elements in crystal-id order.  list keeps
// the developed element list alive for the build.
void build_emulsion_tree(fg_engine* e, const fg_emulsion* em, bool developed_only, RTreeBufs& B,
                         DBuf<uint32_t>& list, bool walks = true);

// fg_develop.cu
void develop(fg_engine* e, fg_emulsion* em, const fg_dev_cfg& cfg, fg_dev_report* rep);

// fg_scan.cu
struct ScanOut {
  float* out = nullptr;      // mode-mapped value per pixel
  uint8_t* image8 = nullptr; // 8-bit image
  float* d_neg = nullptr;    // -log10(clamp(T)) + 0.05
  uint16_t* ray_hits = nullptr;
};
// Host arrays in crystal-id order to and from device arrays in slot order.  The permutation runs on
// the device (a random gather of millions of values costs the host milliseconds; latent counts of 338 k
// crystals read in 50 us, 206 on the host); for few crystals, where its launch and scratch cost more (64: 20 us
// and 14, 9,000: 21 and 20), and where that scratch cannot be allocated, it runs on the host.
constexpr uint32_t PERMUTE_MIN = 8192;
template <class T>
__global__ void k_permute(const T* __restrict__ in, const uint32_t* __restrict__ idx, uint32_t n, T* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[idx[i]];
}
template <class T>
bool permute_scratch(DBuf<T>& b, size_t n, cudaStream_t st) {
  if (n < PERMUTE_MIN) return false;
  try {
    b.alloc(n, st);
  } catch (const Error& x) {
    if (x.st != FG_ERR_OOM) throw;
    (void)cudaGetLastError();
    return false;
  }
  return true;
}
// One such array on its way; it holds host memory of the copy, so it outlives the caller's synchronisation.
template <class T>
class IdCopy {
  std::vector<T> host_;

 public:
  // Enqueues by_id (crystal-id order) to slots (slot order).
  void to_slots(const fg_emulsion* em, const T* by_id, T* slots, cudaStream_t st) {
    const uint32_t n = em->n;
    if (!n) return;
    DBuf<T> tmp;
    if (em->h_s2id.empty()) {
      FG_CUDA(cudaMemcpyAsync(slots, by_id, n * sizeof(T), cudaMemcpyHostToDevice, st));
    } else if (permute_scratch(tmp, n, st)) {
      FG_CUDA(cudaMemcpyAsync(tmp.p, by_id, n * sizeof(T), cudaMemcpyHostToDevice, st));
      k_permute<<<(n + 255) / 256, 256, 0, st>>>(tmp.p, em->sorted_to_id.p, n, slots);
      FG_CUDA(cudaGetLastError());
    } else {
      host_.resize(n);
      for (uint32_t s = 0; s < n; ++s) host_[s] = by_id[em->h_s2id[s]];
      FG_CUDA(cudaMemcpyAsync(slots, host_.data(), n * sizeof(T), cudaMemcpyHostToDevice, st));
    }
  }
  // Enqueues slots to by_id; finish, after the stream was synchronised, puts the last of it in place.
  void from_slots(const fg_emulsion* em, const T* slots, T* by_id, cudaStream_t st) {
    const uint32_t n = em->n;
    if (!n) return;
    DBuf<T> tmp;
    if (em->h_s2id.empty()) {
      FG_CUDA(cudaMemcpyAsync(by_id, slots, n * sizeof(T), cudaMemcpyDeviceToHost, st));
    } else if (permute_scratch(tmp, n, st)) {
      k_permute<<<(n + 255) / 256, 256, 0, st>>>(slots, em->id_to_sorted.p, n, tmp.p);
      FG_CUDA(cudaGetLastError());
      FG_CUDA(cudaMemcpyAsync(by_id, tmp.p, n * sizeof(T), cudaMemcpyDeviceToHost, st));
    } else {
      host_.resize(n);
      FG_CUDA(cudaMemcpyAsync(host_.data(), slots, n * sizeof(T), cudaMemcpyDeviceToHost, st));
    }
  }
  void finish(const fg_emulsion* em, T* by_id) const {
    for (uint32_t s = 0; s < host_.size(); ++s) by_id[em->h_s2id[s]] = host_[s];
  }
};

// fg_image.cu: the separable 3-tap clamp-to-edge filter (two passes through tmp), in the
// reference's FP32 operation order, the second pass scaled by `scale`.
void launch_otf(const float* in, float* tmp, float* out, uint32_t w, uint32_t h, const float k[3], float scale,
                cudaStream_t st);

// Device bytes a batch needs for one tile (fg_batch.cu), a little above what plan() allocates;
// *slots (may be null) receives the tile's crystal slots.
unsigned long long tile_footprint(const fg_tile_params& p, unsigned long long* slots);

// Device state of a new emulsion (counts, development, clumps), zeroed (fg_engine.cu).
void alloc_state(fg_emulsion* em, cudaStream_t st);

// Per-call bookkeeping of the engine entry points (fg_engine.cu): zero the timings and device
// counters; read the counters back, synchronise and raise the device error word.
void begin_call(fg_engine* e);
void end_call(fg_engine* e);
float elapsed(cudaEvent_t a, cudaEvent_t b);

// Strata per axis of a scan's pixels; refuses a size or a number of samples that cannot be scanned.
uint32_t scan_grid(const fg_scan_cfg& cfg);
void scan(fg_engine* e, const fg_emulsion* em, const fg_scan_cfg& cfg, uint64_t seed,
          const float* sigma_sorted, const ScanOut& out);
// g_sorted[s] += sum over the rays of each pixel p of wpx[p] / spp * T_ray * chord_s (device
// arrays; wpx has one weight per pixel, g_sorted one FP64 sum per crystal in Morton order).  T
// receives the transmittance that the forward scan in Negative mode gives.
void scan_adjoint(fg_engine* e, const fg_emulsion* em, const fg_scan_cfg& cfg, uint64_t seed,
                  const float* sigma_sorted, const float* wpx, double* g_sorted, float* T);

// fg_transport.cu
void expose(fg_engine* e, fg_emulsion* em, const float* tile_dev, uint32_t tw, uint32_t th,
            const fg_exposure_cfg& cfg, uint64_t seed, unsigned long long* photons_out);

// Exclusive prefix sum on the device (CUB).
void exclusive_scan_u32(const uint32_t* in, uint32_t* out, size_t n, cudaStream_t st);

// Raises an Error when a kernel reported one through the engine's error word.
void check_error_word(fg_engine* e);

// Runs f under the engine lock with the device current; converts failures to a status.
template <class F>
fg_status guard(fg_engine* e, F&& f) {
  if (!e) return FG_ERR_INVALID_ARG;
  std::lock_guard<std::recursive_mutex> lk(e->mu);
  try {
    FG_CUDA(cudaSetDevice(e->device));
    f();
    return FG_OK;
  } catch (const Error& x) {
    e->err = x.msg;
    return x.st;
  } catch (const std::bad_alloc&) {
    e->err = "host allocation failed";
    return FG_ERR_OOM;
  } catch (const std::exception& x) {
    e->err = x.what();
    return FG_ERR_PIPELINE;
  }
}

inline unsigned grid_for(size_t n, unsigned block) {
  return static_cast<unsigned>((n + block - 1) / block);
}

}  // namespace fg
