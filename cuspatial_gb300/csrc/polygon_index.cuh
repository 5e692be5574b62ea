// Device-resident polygon index used by the point-in-polygon join.
//
// For every polygon the index holds
//   * its vertex bounding box and an anchor (box centre),
//   * each vertex's edge (previous vertex -> vertex, ring-cyclic) as float32
//     offsets from the anchor, plus the largest offset magnitude,
//   * a partition of [ymin, ymax) into slabs, each listing the edges whose
//     y-range (widened by a margin) meets the slab,
//   * the sorted x values of its exactly vertical edges.
//
// Why this is exact against the reference's ring walk
// (detail/algorithm/is_point_in_polygon.cuh:45-100):
//   1. For coordinates of normal magnitude, float_equal(b - a, 0) holds only
//      for b == a, and equality is transitive, so the reference's skipped
//      vertices are exactly those equal to their predecessor and its edges
//      are (p[i-1], p[i]) for the other vertices.  Polygons where a vertex
//      difference is non-zero but within 4 ULP of zero (denormal scale) are
//      flagged and always walked with the reference loop.
//   2. The result is "no on-edge hit" AND the XOR of per-edge toggles, so the
//      edges can be visited in any order and any subset that contains every
//      edge able to toggle or to hit is enough.
//   3. A point with py outside [ymin, ymax) sees equal y-flags on every edge:
//      no toggle, result false.
//   4. An edge toggles only if its y-range contains py; a non-vertical edge
//      can be "collinear and within x-range" only if py lies within
//      2^-48 * |rise| of its y-range.  Each edge is binned over its y-range
//      widened by 2^-36 of its height, which covers both.
//   5. An exactly vertical edge reports "on edge" for any py whenever
//      px == its x (x-range check only, is_point_in_polygon.cuh:75-83); that
//      case is caught by a lookup in the sorted vertical-x list.
//   6. Slab coordinates are float32 roundings of the float64 (y - ymin) *
//      inv_h (2.5e-4 slab at most); edges are further widened by 1/32 of a
//      slab, which covers that and the float32 slab lookup of the filter
//      (below 1e-2 slab under its guard), so every lookup finds every edge.
//
// Anchors lie on a power-of-two grid (2^(e-22) for coordinates below 2^e), so
// the offset between a polygon anchor and a leaf anchor on the same grid is
// exact in float64 and, when below 2^24 grid steps, in float32.
#pragma once

#include <memory>

#include "common.cuh"

namespace cspt {

// x-bins per slab of the float32 index (window records per slab)
constexpr int kSlabBins = 8;
// slab entries: vertex id in bits 0-30, bit 31 set when the edge crosses the
// whole slab (float32 index)
constexpr uint32_t kEntryCrossing = 1u << 31;
constexpr uint32_t kEntryVertex   = kEntryCrossing - 1u;

// A double cut to float32 on the integer pipe: mantissa truncated; below
// float32's normal range -> 0, beyond it or non-finite -> infinity.  Within
// 2^-23 |v| (1.2e-38 below the normal range) of v, toward zero.
__device__ inline float truncated_f32(double v)
{
  unsigned long long const b = static_cast<unsigned long long>(__double_as_longlong(v));
  uint32_t const sign        = static_cast<uint32_t>(b >> 32) & 0x80000000u;
  int const e                = static_cast<int>((b >> 52) & 0x7FFull) - 1023 + 127;
  if (e <= 0) return __uint_as_float(sign);
  if (e >= 255) return __uint_as_float(sign | 0x7F800000u);
  return __uint_as_float(sign | (static_cast<uint32_t>(e) << 23) |
                         static_cast<uint32_t>((b >> 29) & 0x7FFFFFull));
}
// The width that a truncated value t is widened by on both sides: twice its
// truncation error, so that the value itself lies inside by at least
// 2^-23 |t| (not a number for an infinite t: its comparisons decide nothing).
__device__ inline float outward_width(float t)
{
  return __fmaf_ru(fabsf(t), 2.384185791015625e-07f, 1.0e-37f);
}
// The box (xmin, ymin, xmax, ymax) of two points given truncated, wider than
// them by 2^-23 of the larger magnitude on each side, which is more than 2^-24 of
// the difference of their coordinates; the whole plane when a coordinate is
// beyond float32 or not finite.
__device__ inline float4 outward_box(float x0, float y0, float x1, float y1)
{
  float const mx = fmaxf(fabsf(x0), fabsf(x1)), my = fmaxf(fabsf(y0), fabsf(y1));
  float const wx = outward_width(mx), wy = outward_width(my);
  if (!(wx < INFINITY && wy < INFINITY))
    return make_float4(-INFINITY, -INFINITY, INFINITY, INFINITY);
  return make_float4(__fsub_rd(fminf(x0, x1), wx), __fsub_rd(fminf(y0, y1), wy),
                     __fadd_ru(fmaxf(x0, x1), wx), __fadd_ru(fmaxf(y0, y1), wy));
}

// Whether an index that leaves the choice to the device carries edge bounds
// (place: the view's origin).
template <typename T>
__device__ inline bool has_bounds(T const* place, T bounds_share)
{
  return place[2] >= bounds_share && place[3] >= bounds_share;
}

template <typename T>
struct PolygonIndexView {
  // polygon topology (caller's arrays)
  uint32_t const* poly_offsets;
  uint32_t const* ring_offsets;
  T const* vx;
  T const* vy;
  size_t num_polygons;
  // per polygon
  T const* pminx;
  T const* pminy;
  T const* pmaxx;
  T const* pmaxy;
  T const* anchor_x;           // box centre rounded to the grid
  T const* anchor_y;
  T const* grid;               // device scalar: the anchor grid step
  T const* origin;             // x and y that edge bounds are relative to, and the share
                               // of the common box that the median polygon's takes
  long long const* anchor_ix;  // anchors in grid steps
  long long const* anchor_iy;
  float const* inv_slab_h32;   // inv_slab_h rounded to float
  T const* inv_slab_h;         // slabs per unit of y
  float const* max_offset;     // largest |float32 offset| over the polygon's vertices
  float4 const* box32;         // vertex box as float32 offsets from the anchor
                               // (edge bounds: the vertex box from the origin, outward)
  uint32_t const* num_slabs;
  uint32_t const* slab_base;   // first slab of the polygon in slab_start
  uint8_t const* exact_only;   // 1: walk the reference loop, no index
  uint32_t const* vert_begin;  // sorted vertical-edge x values, per polygon range
  uint32_t const* vert_end;
  T const* vert_x;
  float const* vert_x32;
  // per slab: entries [slab_start[s], slab_start[s+1])
  uint32_t const* slab_start;
  uint32_t const* slab_edges;  // vertex index of the edge's end point | kEntryCrossing
  float4 const* slab_e32;      // the entry's edge (ax, ay, bx, by) as float32 offsets
                               // (edge bounds: its box from the origin, outward_box)
  // per vertex
  uint32_t const* prev_vertex;
  float4 const* edge32;        // (ax, ay, bx, by) offsets from the anchor
                               // (edge bounds: from the origin, truncated)
  // float32 index: per slab, the entries crossing the whole slab come first
  // (sorted left to right); per (slab, x-bin) a window record
  // lo | hi << 15 | parity << 30 (see slab_order_kernel)
  uint32_t const* slab_nfull;  // null: slabs not ordered
  uint32_t const* slab_bins;
  float const* inv_bin_w32;    // x-bins per unit of x (0: no bins)
};

template <typename T>
class PolygonIndex {
 public:
  // order_slabs (float32 index only): sort each slab's crossing edges and
  // build the per-(slab, x-bin) windows.  It costs a pass over all slab
  // entries and pays off where the index is evaluated many times (batched
  // plans, resident polygon sets).
  // edge_bounds (float64 index): slab entries carry their edge's box in float32,
  // rounded outward (outward_box), in place of the float32 edges.  With
  // build_float32 too, the device decides: bounds where the median polygon takes at
  // least bounds_share of the common box along both axes, else float32 edges; the
  // kernels of both kinds are launched and ask has_bounds.
  // defer_fill: return once the per-polygon boxes, slab counts and the anchor
  // grid are enqueued (array sizes come from bounds on the host, so the call
  // does not wait for the device); fill() then writes the slab entries.  Work
  // that needs only grid() can run on another stream meanwhile, once it waits
  // for the calling stream.
  PolygonIndex(uint32_t const* poly_offsets, size_t num_poly_offsets,
               uint32_t const* ring_offsets, size_t num_ring_offsets, T const* vx, T const* vy,
               size_t num_vertices, bool build_float32, Allocator const& alloc,
               bool order_slabs = false, bool defer_fill = false, bool edge_bounds = false,
               T bounds_share = T{0});
  ~PolygonIndex();
  PolygonIndex(PolygonIndex const&)            = delete;
  PolygonIndex& operator=(PolygonIndex const&) = delete;
  void fill();
  // device scalar: the anchor grid step (valid before fill())
  T const* grid() const { return grid_.data(); }
  // device: x and y of the edge bounds' origin (valid before fill())
  T const* origin() const { return grid_.data() + 1; }
  PolygonIndexView<T> view() const { return v_; }
  bool edge_bounds() const { return edge_bounds_; }

 private:
  struct Sizing;  // state carried from the sizing pass to fill()
  std::unique_ptr<Sizing> sizing_;
  bool edge_bounds_ = false;
  Buffer<T> pminx_, pminy_, pmaxx_, pmaxy_, ax_, ay_, invh_, vert_x_, grid_;
  Buffer<float> maxoff_, vert_x32_, invh32_;
  Buffer<long long> aix_, aiy_;
  Buffer<uint32_t> nslab_, slab_base_, vbeg_, vend_, slab_start_, slab_edges_, prev_;
  Buffer<uint8_t> exact_;
  Buffer<float4> edge32_, box32_, slab_e32_;
  Buffer<uint32_t> slab_nfull_, slab_bins_;
  Buffer<float> invw32_;
  PolygonIndexView<T> v_{};
};

// A planned float64 point-in-polygon evaluation (defined in pip.cu).
class PipExec {
 public:
  PipExec(uint32_t const* pair_poly, uint32_t const* pair_quad, size_t npairs,
          uint32_t const* qlen, uint32_t const* qoff, uint32_t const* point_indices, size_t npi,
          double const* x, double const* y, PolygonIndexView<double> const& ix, bool filtered,
          unsigned block_threads, Allocator const& alloc);
  ~PipExec();
  PipExec(PipExec const&)            = delete;
  PipExec& operator=(PipExec const&) = delete;
  void execute(cudaStream_t s, uint32_t* out_poly, uint32_t* out_point, uint64_t cap);
  void evaluate(cudaStream_t s);  // bits, counts and output offsets
  void expand(cudaStream_t s, uint32_t* out_poly, uint32_t* out_point, uint64_t cap);
  uint64_t const* total() const;             // device: number of output pairs
  uint64_t const* pair_out_offsets() const;  // device: first output of each pair
  int const* overflow() const;               // device: 1 when total > cap
  unsigned long long const* refined() const;

 private:
  class Impl;
  Impl* impl_;
};

}  // namespace cspt
