// Fused box-image kernels: per test point, box centre -> grid point -> map -> depth-d
// code -> leaf index, all in FP64 registers.  This is the reference's
// GridPointsFunctor (Functors.hpp:476-511) consumed by thrust::lower_bound and
// ComputeSearchIndexFunctor (ImplicitBoxTree.hpp:2394-2432), evaluated once per point
// instead of twice and without the point stream ever being stored.
#include <type_traits>

#include "kernels.h"
#include "rows.cuh"

namespace b12g {

namespace {

constexpr int kThreads = 256;

// the source box of point (rank, k) and the leaf index its image lands in
template<class Map, class Grid>
struct PointImage {
  static constexpr int D = Map::D;

  // per-dimension indices of source box `leaf` at a.depth (in children mode: child
  // leaf & 1 of leaf leaf >> 1): from the packed keys the lookup table was built from,
  // else from the code
  static __device__ __forceinline__ void source_bits(const ImageArgs& a, uint32_t leaf, uint32_t (&bits)[D])
  {
    if (a.hash.pk) {
      if (a.children) {
        unpack_bits_k<D>(__ldg(a.hash.pk + (leaf >> 1)), a.dc.kp, bits);
        const int jd = a.dc.jd;                    // the last bisection splits dimension jd
#pragma unroll
        for (int j = 0; j < D; ++j)                // (no dynamic index: the array stays in registers)
          if (j == jd) bits[j] = (bits[j] << 1) | (leaf & 1u);
      } else {
        unpack_bits_k<D>(__ldg(a.hash.pk + leaf), a.dc.k, bits);
      }
      return;
    }
    const uint64_t code =
        a.children ? ((__ldg(a.codes + (leaf >> 1)) << 1) | uint64_t(leaf & 1u)) : __ldg(a.codes + leaf);
#pragma unroll
    for (int j = 0; j < D; ++j) bits[j] = deinterleave<D>(code, a.depth, j);
  }

  // grid point k of a box (point i of the launch).  `pts` is the block's grid-point table
  // (dimension-major, P entries per dimension) when the grid has one, else the 1-D
  // coordinate table.
  static __device__ __forceinline__ void grid_point(const ImageArgs& a, const double* pts, bool use_table, uint64_t i,
                                                    uint32_t k, double (&g)[D])
  {
    if (Grid::kTable && use_table) {
#pragma unroll
      for (int j = 0; j < D; ++j) g[j] = pts[j * uint32_t(a.points) + k];
    } else {
      Grid::template point<D>(a.grid, pts, i, k, g);
    }
  }

  // returns whether the image point lies in the domain; `tbits` its box's per-dimension
  // indices at a.depth; from the source box's centre (its radius is the launch's).
  // kCold: the evaluation of the few points that a screened launch could not decide
  template<bool kCold = false>
  static __device__ __forceinline__ bool image_at(const ImageArgs& a, const double* pts, bool use_table,
                                                  const double (&c)[D], uint64_t i, uint32_t k, uint32_t (&tbits)[D])
  {
    double g[D], x[D], y[D];
    grid_point(a, pts, use_table, i, k, g);
#pragma unroll
    for (int j = 0; j < D; ++j) x[j] = __dadd_rn(c[j], __dmul_rn(g[j], a.dc.ax[j].rk));
    if constexpr (kCold) Map::apply_cold(a.map, x, y);
    else Map::apply(a.map, x, y);
    return point_bits<D>(a.dom, a.dc, y, tbits);
  }

  // the same from the source box's indices
  template<bool kCold = false>
  static __device__ __forceinline__ bool image(const ImageArgs& a, const double* pts, bool use_table,
                                               const uint32_t (&sbits)[D], uint64_t i, uint32_t k,
                                               uint32_t (&tbits)[D])
  {
    double c[D], r;
#pragma unroll
    for (int j = 0; j < D; ++j) box_axis(a.dom, a.dc.ax[j], j, sbits[j], c[j], r);
    return image_at<kCold>(a, pts, use_table, c, i, k, tbits);
  }

  // the screened evaluation from the source box's indices: whether it decided the point
  static __device__ __forceinline__ bool screened(const ImageArgs& a, const double* pts, bool use_table,
                                                  const uint32_t (&sbits)[D], uint64_t i, uint32_t k,
                                                  uint32_t (&tbits)[D], bool& valid)
  {
    double g[D], x[D];
    grid_point(a, pts, use_table, i, k, g);
#pragma unroll
    for (int j = 0; j < D; ++j)
      x[j] = __fma_rn(g[j], a.sc.sR[j], __fma_rn(screen_index(sbits[j], a.sc.bits[j]), a.sc.sA[j], a.sc.sB[j]));
    const bool kept = Screen<Map>::run(a.sc, a.map, x);
    return screen_locate<D>(a.sc, x, tbits, valid) && kept;
  }

  // the same from its centre
  static __device__ __forceinline__ bool screened_at(const ImageArgs& a, const double* pts, bool use_table,
                                                     const double (&c)[D], uint64_t i, uint32_t k,
                                                     uint32_t (&tbits)[D], bool& valid)
  {
    double g[D], x[D];
    if constexpr (std::is_same<Grid, PhiloxGrid>::value) {
      Grid::template raised<D>(a.grid, i, g);
#pragma unroll
      for (int j = 0; j < D; ++j) x[j] = __fma_rn(g[j], a.sc.sR[j], __fma_rn(c[j], a.sc.sC[j], a.sc.sP[j]));
    } else {
      grid_point(a, pts, use_table, i, k, g);
#pragma unroll
      for (int j = 0; j < D; ++j) x[j] = __fma_rn(g[j], a.sc.sR[j], __fma_rn(c[j], a.sc.sC[j], a.sc.sD[j]));
    }
    const bool kept = Screen<Map>::run(a.sc, a.map, x);
    return screen_locate<D>(a.sc, x, tbits, valid) && kept;
  }

  // centre of source `rank` from the launch's table
  static __device__ __forceinline__ void source_centre(const ImageArgs& a, uint64_t rank, double (&c)[D])
  {
    const double2* p = reinterpret_cast<const double2*>(a.src_c + kSrcStride * rank);
    const double2 c01 = __ldg(p);
    c[0] = c01.x;
    if (D > 1) c[D > 1 ? 1 : 0] = c01.y;
    if (D > 2) {
      const double2 c23 = __ldg(p + 1);
      c[D > 2 ? 2 : 0] = c23.x;
      if (D > 3) c[D > 3 ? 3 : 0] = c23.y;
    }
  }

  static __device__ __forceinline__ uint32_t target(const ImageArgs& a, uint32_t n, bool valid,
                                                    const uint32_t (&tbits)[D])
  {
    if (!a.children) return find_leaf_bits<D>(a.hash, a.codes, n, valid, tbits, a.depth, a.dc.k);
    if (!valid) return kInvalidIndex;
    const int jd = a.dc.jd;
    uint32_t pbits[D], child = 0;
#pragma unroll
    for (int j = 0; j < D; ++j) {
      pbits[j] = j == jd ? tbits[j] >> 1 : tbits[j];
      if (j == jd) child = tbits[j] & 1u;
    }
    const uint32_t p = find_leaf_bits<D>(a.hash, a.codes, n, true, pbits, a.depth - 1, a.dc.kp);
    return p == kInvalidIndex ? kInvalidIndex : 2u * p + child;
  }
};

constexpr uint32_t kPointTable = 2048;  // doubles of grid-point table per block (16 KB)
constexpr int kChunkTrips = 4;          // units (a point a lane) a warp takes at a time from the work queue;
                                        // twice as many in Mark mode, whose points are short and whose
                                        // launches large (the continuation 9.27 ms, with four 9.46)
constexpr int kFineUnits = 4;           // units a warp left in the queue when it takes single ones: more suit a
                                        // forced Duffing job's small launches (1, 4 and 8 in ratio: 1.11, 1,
                                        // 0.98), fewer the continuation's large ones (0.995, 1, 1.03)

// fills `pts` with the P x D grid points when they fit (returns true), else with the
// 1-D coordinates for the per-point path
template<class Grid, int D>
__device__ __forceinline__ bool load_points(const GridParams& g, uint64_t P, double* pts)
{
  const bool table = Grid::kTable && P * D <= kPointTable;
  if (table) {
    for (uint32_t idx = threadIdx.x; idx < uint32_t(P) * D; idx += blockDim.x) {
      const int j = int(idx / uint32_t(P));
      pts[idx] = Grid::table_value(g, g.coord, idx - uint32_t(j) * uint32_t(P), j);
    }
  } else {
    for (uint32_t i = threadIdx.x; i < 64; i += blockDim.x) pts[i] = g.coord[i];
  }
  __syncthreads();
  return table;
}

// Bound by instruction issue: an FP64 instruction holds its scheduler for two cycles and
// any other for one.  kScreen: the screened evaluation (screen.cuh), 736 FP64 and about 310
// other instructions per 32 Lorenz points against 942 and 290 (FMA) or 1,600 (strict); the
// image launches of a depth-27 job take 5.52 ms against 6.58 (FMA) and 10.21 (strict).  Four
// blocks an SM, 64 registers: the coefficients stay in registers over the unrolled steps
// (five blocks with 48: 5.72 ms, three: 5.52).  Mark mode (the continuation, short points):
// five blocks, 9.27 ms, 2 % less than with four.
template<class Map, class Grid, ImageMode M, bool kScreen>
__global__ void __launch_bounds__(kThreads, !kScreen ? 6 : M == ImageMode::Mark ? 5 : 4) image_points_kernel(const ImageArgs a)
{
  using PI = PointImage<Map, Grid>;
  __shared__ double pts[kPointTable];
  const uint32_t n = *a.n_leaves;
  const uint32_t nboxes = M == ImageMode::Mark ? a.n_src_value : a.n_src ? *a.n_src : (a.children ? 2u * n : n);
  const uint64_t P = a.points;
  const uint32_t P32 = uint32_t(P);
  const uint64_t total = uint64_t(nboxes) * P;
  const int lane = threadIdx.x & 31;
  // the queue of the next launch on the tree's stream starts empty
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.work_next = 0u;
  if (M == ImageMode::Hit && a.children && 2ull * n > a.hit_cap) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(a.error, 1u);
    return;
  }
  // A device work queue (UnitQueue) of 32-point units (of 2^shift times as many where that
  // many units would not fit 32 bits): every warp takes the next points until none is left,
  // so that warps that run faster do more (a static grid-stride split left the slower warps
  // alone at the end: 47 % of the warp slots were active on average, of 75 % possible).
  constexpr uint32_t kTake = M == ImageMode::Mark ? 2 * kChunkTrips : kChunkTrips;
  uint32_t shift = 0;
  while (((total + 31) >> (5 + shift)) >= 0x40000000ull) ++shift;
  UnitQueue<kTake, kFineUnits, M != ImageMode::Mark> q(a.work, uint32_t((total + (32ull << shift) - 1) >> (5 + shift)));
  if (q.idle_block()) return;
  // Mark mode: an index's place in the box's code, by dimension, where the indices have at
  // most 8 bits (four reads and two ORs instead of 36 instructions of bit spreading)
  __shared__ uint32_t spread[M == ImageMode::Mark ? Map::D * 256 : 1];
  bool spread_ok = false;
  if constexpr (M == ImageMode::Mark) {
    spread_ok = a.dc.c32 && a.dc.k[0] <= 8;
    if (spread_ok)
      for (uint32_t i = threadIdx.x; i < Map::D * 256; i += blockDim.x) {
        uint32_t one[Map::D] = {};
        one[i >> 8] = i & 255u;
        spread[i] = uint32_t(code_of_bits<Map::D>(a.dc, one, a.depth));
      }
  }
  const bool table = load_points<Grid, Map::D>(a.grid, a.points, pts);   // (ends with a block barrier)

  // Mark mode: the warp's new boxes (the same in every lane), added to the launch's count at
  // the end (an atomic for every warp with a new box cost the continuation's image launches
  // an eighth of their time)
  uint32_t new_boxes = 0;
  // (the coupled Duffing continuation always tries: its points are short and few of them stay
  // undecided; 10.68 ms, with the trial 10.85)
  constexpr bool kTrial = kScreen && !(M == ImageMode::Mark && Map::D == 4);
  ScreenTrial trial;
  uint32_t undecided = 0;
  // One point of the launch: g = rank * P + k (the source's rank among the sources, the
  // point's index in its box).  Every lane of the warp calls it the same number of times
  // (inactive lanes with active = false), so that the warp collectives stay converged.
  auto point = [&](uint64_t g, uint32_t rank, uint32_t k, bool active) {
    uint32_t t = kInvalidIndex;
    uint32_t tbits[Map::D];
    bool valid = false, sure = true;
    if (active) {
      if constexpr (M == ImageMode::Insert || M == ImageMode::Mark) {   // these carry their source centres
        double c[Map::D];
        PI::source_centre(a, rank, c);
        if constexpr (kScreen) {
          sure = (!kTrial || trial.on()) && PI::screened_at(a, pts, table, c, g, k, tbits, valid);
          if (!sure) {
            valid = PI::template image_at<true>(a, pts, table, c, g, k, tbits);
            ++undecided;
          }
        } else {
          valid = PI::image_at(a, pts, table, c, g, k, tbits);
        }
      } else {
        const uint32_t leaf = a.src ? __ldg(a.src + rank) : uint32_t(rank);
        uint32_t sbits[Map::D];
        PI::source_bits(a, leaf, sbits);
        if constexpr (kScreen) {
          sure = (!kTrial || trial.on()) && PI::screened(a, pts, table, sbits, g, k, tbits, valid);
          if (!sure) {
            ++undecided;
            PI::source_bits(a, leaf, sbits);       // (read again: not kept over the evaluation)
            valid = PI::template image<true>(a, pts, table, sbits, g, k, tbits);
          }
        } else {
          valid = PI::image(a, pts, table, sbits, g, k, tbits);
        }
      }
      if constexpr (M != ImageMode::Mark) t = PI::target(a, n, valid, tbits);
    }
    if constexpr (kTrial && ScreenTrial::by_unit(Map::D)) trial.note(!sure, 1);
    if constexpr (M == ImageMode::Hit) {
      // (a store of all lanes: the warp's few distinct bytes leave the SM as so many sectors
      // either way, and finding one lane for each cost more than it saved)
      if (t != kInvalidIndex) a.hit[t] = 1;
      if (a.targets && active) {
        if (g < a.targets_cap) a.targets[g] = valid ? t : kOutsideIndex;
        else *a.targets_over = 1;
      }
    } else if constexpr (M == ImageMode::Search) {
      if (active) a.out[g] = t;
    } else if constexpr (M == ImageMode::Mark) {
      // the image's box, unless its bit is set already (a stale read only sends the point
      // on to the atomic), deduplicated within the warp: most warps find no new box.  The lane
      // whose atomic sets the bit marks the box in `fresh`.
      uint32_t code = 0;
      bool fresh = false;
      if (active && valid) {
        if (spread_ok) {
          code = 0;
#pragma unroll
          for (int j = 0; j < Map::D; ++j) code |= spread[j * 256 + tbits[j]];
        } else {
          code = uint32_t(code_of_bits<Map::D>(a.dc, tbits, a.depth));
        }
        fresh = !((a.bits[code >> 5] >> (code & 31u)) & 1u);
      }
      if (__any_sync(0xFFFFFFFFu, fresh)) {
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, fresh ? code : ~0u) & __ballot_sync(0xFFFFFFFFu, fresh);
        fresh = fresh && lane == __ffs(peers) - 1;
        if (fresh) {
          const uint32_t m = 1u << (code & 31u);
          fresh = !(atomicOr(a.bits + (code >> 5), m) & m);
          if (fresh) atomicOr(a.fresh + (code >> 5), m);
        }
        const unsigned lead_mask = __ballot_sync(0xFFFFFFFFu, fresh);
        new_boxes += uint32_t(__popc(lead_mask));
      }
    } else {
      // candidates: valid images that are not leaves, as packed keys (the caller turns them
      // into codes); deduplicated within the warp and appended with one atomic per warp
      if (a.hit) {
        const unsigned hp = __match_any_sync(0xFFFFFFFFu, t);
        if (active && t != kInvalidIndex && lane == __ffs(hp) - 1) a.hit[t] = 1;
      }
      const bool is_cand = active && valid && t == kInvalidIndex;
      const uint64_t tcode = is_cand ? pack_bits_k<Map::D>(tbits, a.dc.k) : 0ull;
      const uint64_t key = is_cand ? tcode : kInvalidCode;
      // (the lowest candidate lane of each key leads: a non-candidate lane may share the
      // all-ones key)
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, key) & __ballot_sync(0xFFFFFFFFu, is_cand);
      bool leader = is_cand && lane == __ffs(peers) - 1;
      if (a.claim && leader) leader = hash_claim(a.hash, tcode, a.error);
      const unsigned lead_mask = __ballot_sync(0xFFFFFFFFu, leader);
      uint32_t slot = 0;
      if (lane == 0 && lead_mask) slot = atomicAdd(a.cand_count, uint32_t(__popc(lead_mask)));
      slot = __shfl_sync(0xFFFFFFFFu, slot, 0);
      if (leader) {
        const uint32_t pos = slot + __popc(lead_mask & ((1u << lane) - 1u));
        if (pos < a.cand_cap) a.cand[pos] = tcode;
        else atomicOr(a.error, 1u);
      }
    }
  };

  for (bool more = q.any(); more; more = q.next()) {
    const uint32_t c = q.at, size = q.size;
    // (sources and points per box both fit 32 bits: the rank and the point index do)
    const uint64_t g = (uint64_t(c) << (5 + shift)) + uint64_t(lane);
    uint32_t rank, k;
    if (total <= 0xFFFFFFFFull - 64ull * kTake) {
      rank = uint32_t(g) / P32;
      k = uint32_t(g) - rank * P32;
    } else {
      rank = uint32_t(g / P);
      k = uint32_t(g - uint64_t(rank) * P);
    }
#pragma unroll 1
    for (uint32_t j = 0; j < (size << shift); ++j) {
      const uint64_t gj = g + 32ull * uint64_t(j);
      point(gj, rank, k, gj < total);
      k += 32;
      while (k >= P32) { k -= P32; ++rank; }
    }
    if constexpr (kTrial && !ScreenTrial::by_unit(Map::D)) {
      trial.note(undecided, size << shift);
      undecided = 0;
    }
  }
  if constexpr (M == ImageMode::Mark) {
    if (lane == 0 && new_boxes) atomicAdd(a.cand_count, new_boxes);
  }
}

// ---------------------------------------------------------------------------------
// transition rows: warp per source box; the box's P <= 128 targets are sorted in
// shared memory and run-length counted, giving the row's (column, count) pairs in
// column order - the reference's packed (row, col) radix sort plus reverse
// inclusive_scan_by_key and unique_by_key (ImplicitBoxTree.hpp:3007-3038) done per row
// ---------------------------------------------------------------------------------
constexpr int kRowWarps = kThreads / 32;

// (registers: three blocks an SM for Lorenz, four for the others)
template<class Map, class Grid, bool kScreen>
__global__ void __launch_bounds__(kThreads, !kScreen ? 1 : Map::D == 3 ? 3 : 4) transition_rows_kernel(const RowArgs ra)
{
  using PI = PointImage<Map, Grid>;
  const ImageArgs& a = ra.img;
  __shared__ double pts[kPointTable];
  __shared__ uint32_t keys[kRowWarps][128];
  __shared__ uint32_t bounds[kRowWarps][4];
  const bool table = load_points<Grid, Map::D>(a.grid, a.points, pts);

  const uint32_t n = *a.n_leaves;
  const uint32_t nrows = a.n_src ? *a.n_src : n;
  const uint32_t P = uint32_t(a.points);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t* s = keys[w];
  const uint32_t warps = gridDim.x * kRowWarps;
  ScreenTrial trial;

  for (uint32_t row = blockIdx.x * kRowWarps + w; row < nrows; row += warps) {
    const uint32_t leaf = a.src ? __ldg(a.src + row) : row;
    uint32_t sbits[Map::D];
    PI::source_bits(a, leaf, sbits);
    uint32_t undecided = 0;
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      const uint32_t k = uint32_t(lane) + 32u * q;
      uint32_t key = kPadKey;
      bool sure = true;
      if (k < P) {
        uint32_t tbits[Map::D];
        const uint64_t i = uint64_t(row) * P + k;
        bool valid;
        if constexpr (kScreen) {
          sure = trial.on() && PI::screened(a, pts, table, sbits, i, k, tbits, valid);
          if (!sure) valid = PI::template image<true>(a, pts, table, sbits, i, k, tbits);
        } else {
          valid = PI::image(a, pts, table, sbits, i, k, tbits);
        }
        const uint32_t t = PI::target(a, n, valid, tbits);
        key = t == kInvalidIndex ? kLostKey : t;
      }
      if (kScreen && !sure) ++undecided;
      s[lane + 32 * q] = key;
    }
    if constexpr (kScreen) trial.note(undecided, (P + 31u) / 32u);
    const uint32_t total = row_emit(s, bounds[w], lane, P, ra.keep_lost, ra.lost_col,
                                    ra.stage_col + size_t(row) * P, ra.stage_cnt + size_t(row) * P);
    if (lane == 0) ra.row_count[row] = total;
    __syncwarp();
  }
}

template<class Map, class Grid, ImageMode M, bool kScreen>
cudaError_t launch_image_mode(const ImageArgs& a, uint64_t max_points, cudaStream_t s)
{
  static int blocks_per_sm = 0;
  if (!blocks_per_sm) {
    int b = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, image_points_kernel<Map, Grid, M, kScreen>, kThreads, 0);
    blocks_per_sm = b > 0 ? b : 1;
  }
  const uint64_t want = (max_points + kThreads - 1) / kThreads;
  const uint64_t cap = uint64_t(device_sm_count()) * blocks_per_sm;
  const unsigned grid = unsigned(want < 1 ? 1 : (want < cap ? want : cap));
  image_points_kernel<Map, Grid, M, kScreen><<<grid, kThreads, 0, s>>>(a);
  return cudaGetLastError();
}

template<class Map, class Grid, bool kScreen>
cudaError_t launch_image_t(ImageMode mode, const ImageArgs& a, uint64_t max_points, cudaStream_t s)
{
  switch (mode) {
    case ImageMode::Hit: return launch_image_mode<Map, Grid, ImageMode::Hit, kScreen>(a, max_points, s);
    case ImageMode::Search: return launch_image_mode<Map, Grid, ImageMode::Search, kScreen>(a, max_points, s);
    case ImageMode::Insert: return launch_image_mode<Map, Grid, ImageMode::Insert, kScreen>(a, max_points, s);
    default: return launch_image_mode<Map, Grid, ImageMode::Mark, kScreen>(a, max_points, s);
  }
}

template<class Map, class Grid, bool kScreen>
cudaError_t launch_rows_t(const RowArgs& a, uint32_t max_rows, cudaStream_t s)
{
  static int blocks_per_sm = 0;
  if (!blocks_per_sm) {
    int b = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, transition_rows_kernel<Map, Grid, kScreen>, kThreads, 0);
    blocks_per_sm = b > 0 ? b : 1;
  }
  const uint64_t want = (uint64_t(max_rows) + kRowWarps - 1) / kRowWarps;
  const uint64_t cap = uint64_t(device_sm_count()) * blocks_per_sm;
  const unsigned grid = unsigned(want < 1 ? 1 : (want < cap ? want : cap));
  transition_rows_kernel<Map, Grid, kScreen><<<grid, kThreads, 0, s>>>(a);
  return cudaGetLastError();
}

// (map, arith, grid) dispatch; each map has a fixed dimension
template<class F>
cudaError_t dispatch(uint32_t map_kind, uint32_t arith, uint32_t grid_kind, uint32_t dim, F&& f)
{
  auto with_grid = [&](auto map_tag) -> cudaError_t {
    using Map = decltype(map_tag);
    if (dim != uint32_t(Map::D)) return cudaErrorInvalidValue;
    switch (grid_kind) {
      case B12G_GRID_INNER: return f(Map{}, InnerGrid{});
      case B12G_GRID_FULL: return f(Map{}, FullGrid{});
      case B12G_GRID_PHILOX: return f(Map{}, PhiloxGrid{});
      default: return cudaErrorInvalidValue;
    }
  };
  switch (map_kind) {
    case B12G_MAP_HENON: return arith == B12G_ARITH_STRICT ? with_grid(HenonMap{}) : cudaErrorInvalidValue;
    case B12G_MAP_LORENZ:
      return arith == B12G_ARITH_FMA ? with_grid(LorenzMap<Fused>{}) : with_grid(LorenzMap<Strict>{});
    case B12G_MAP_COUPLED_DUFFING:
      return arith == B12G_ARITH_STRICT ? with_grid(CoupledDuffingMap{}) : cudaErrorInvalidValue;
    case B12G_MAP_FORCED_DUFFING:
      return arith == B12G_ARITH_STRICT ? with_grid(ForcedDuffingMap{}) : cudaErrorInvalidValue;
    default: return cudaErrorInvalidValue;
  }
}

// a warp per child of the step that stored the targets: the child is a row when it
// survived (its rank advances); a target is a column when its child survived, at the
// child's rank; a point that left the domain is found in a last leaf of code 0
__global__ void __launch_bounds__(kThreads) stored_rows_kernel(const StoredRowArgs a)
{
  __shared__ uint32_t keys[kRowWarps][128];
  __shared__ uint32_t bounds[kRowWarps][4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t* s = keys[w];
  const uint32_t P = a.points, n = a.n_leaves;
  const bool zero_leaf = n > 0 && __ldg(a.codes + n - 1) == 0;
  for (uint32_t c = blockIdx.x * kRowWarps + w; c < a.n_children; c += gridDim.x * kRowWarps) {
    const uint32_t row = __ldg(a.rank + c);
    if (__ldg(a.rank + c + 1) == row) continue;        // removed: no row (warp-uniform)
    // every load of the row goes out before any is used: the targets, then their ranks
    uint32_t tg[4], lo[4], hi[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t k = uint32_t(lane) + 32u * q;
      tg[q] = k < P ? __ldg(a.targets + size_t(c) * P + k) : kInvalidIndex;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const bool in = tg[q] < kOutsideIndex;
      lo[q] = in ? __ldg(a.rank + tg[q]) : 0u;
      hi[q] = in ? __ldg(a.rank + tg[q] + 1) : 0u;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t k = uint32_t(lane) + 32u * q, t = tg[q];
      uint32_t key = kPadKey;
      if (k < P) {
        if (t < kOutsideIndex) key = hi[q] != lo[q] ? lo[q] : kLostKey;
        else key = (t == kOutsideIndex && zero_leaf) ? n - 1 : kLostKey;
      }
      s[lane + 32 * q] = key;
    }
    const uint32_t total = row_emit(s, bounds[w], lane, P, a.keep_lost, n + 1, a.stage_col + size_t(row) * P,
                                    a.stage_cnt + size_t(row) * P);
    if (lane == 0) a.row_count[row] = total;
    __syncwarp();
  }
}

}  // namespace

cudaError_t launch_stored_rows(const StoredRowArgs& a, cudaStream_t s)
{
  if (a.n_children == 0) return cudaSuccess;
  const uint64_t want = (uint64_t(a.n_children) + kRowWarps - 1) / kRowWarps;
  const uint64_t cap = uint64_t(device_sm_count()) * 8;
  stored_rows_kernel<<<unsigned(want < cap ? want : cap), kThreads, 0, s>>>(a);
  return cudaGetLastError();
}

bool image_supported(uint32_t map_kind, uint32_t arith, uint32_t grid_kind, uint32_t dim)
{
  return dispatch(map_kind, arith, grid_kind, dim, [](auto, auto) { return cudaSuccess; }) == cudaSuccess;
}

cudaError_t launch_image(uint32_t map_kind, uint32_t arith, uint32_t grid_kind, uint32_t dim, ImageMode mode,
                         const ImageArgs& a, uint64_t max_points, cudaStream_t s)
{
  if (!a.work || !a.work_turn) return cudaErrorInvalidValue;   // the image kernel takes its points from a work queue
  ImageArgs b = a;
  b.work = a.work + (*a.work_turn & 1u);
  b.work_next = a.work + ((*a.work_turn & 1u) ^ 1u);
  fill_depth_const(b.dom, int(dim), b.depth, b.dc);
  fill_screen(map_kind, b.map, b.dom, int(dim), b.depth, grid_reach(grid_kind, b.grid), b.plan, b.sc);
  return dispatch(map_kind, arith, grid_kind, dim, [&](auto map, auto grid) {
    using Map = decltype(map);
    using Grid = decltype(grid);
    cudaError_t e = cudaErrorInvalidValue;
    if constexpr (Screen<Map>::kOk) {
      if (b.sc.on) e = launch_image_t<Map, Grid, true>(mode, b, max_points, s);
    }
    if (!Screen<Map>::kOk || !b.sc.on) e = launch_image_t<Map, Grid, false>(mode, b, max_points, s);
    if (e == cudaSuccess) *a.work_turn ^= 1u;
    return e;
  });
}

cudaError_t launch_rows(uint32_t map_kind, uint32_t arith, uint32_t grid_kind, uint32_t dim, const RowArgs& a,
                        uint32_t max_rows, cudaStream_t s)
{
  RowArgs b = a;
  fill_depth_const(b.img.dom, int(dim), b.img.depth, b.img.dc);
  fill_screen(map_kind, b.img.map, b.img.dom, int(dim), b.img.depth, grid_reach(grid_kind, b.img.grid), b.img.plan,
              b.img.sc);
  return dispatch(map_kind, arith, grid_kind, dim, [&](auto map, auto grid) {
    using Map = decltype(map);
    using Grid = decltype(grid);
    if constexpr (Screen<Map>::kOk) {
      if (b.img.sc.on) return launch_rows_t<Map, Grid, true>(b, max_rows, s);
    }
    return launch_rows_t<Map, Grid, false>(b, max_rows, s);
  });
}

}  // namespace b12g
