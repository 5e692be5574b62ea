// Quadtree point-to-nearest-linestring join on sm_103a.
//
// Reference: cpp/include/cuspatial/detail/join/quadtree_point_to_nearest_
// linestring.cuh:143-312 and detail/algorithm/point_linestring_distance.cuh:
// 26-51.
//
// The reference enumerates, per quadrant, the (point, linestring) candidates
// point-major (the "transposed" index math at :63-89), reduces each point's
// run with a custom minimum (:279-294) and scatters to the point's position.
// Here the consecutive pairs that share a quadrant form a group; one warp owns
// a group, each lane a point, and the lane folds the group's linestrings in
// pair order with the same rule:
//   a running distance of exactly 0 yields to the next candidate, a new
//   candidate at exactly 0 never wins, equal distances keep the smaller id,
//   otherwise the smaller distance wins.
// The distance is the reference's expression with its dot products contracted
// the way nvcc contracts a.x*b.x + a.y*b.y (one FMA on the x term).
//
// Exact method: linestrings and chunks of segments whose bounding box is
// certainly farther than the running winner are passed over (box_lower); the
// distances that decide are the reference's expression in the input type.
//
// Filtered method (float64 inputs): each segment is first bounded in float32
// with a forward error bound; only segments whose lower bound can still beat
// the best upper bound of the point are evaluated with the float64
// expression, so the winner and its distance are the exact ones.
#include <algorithm>
#include <memory>

#include "common.cuh"
#include "leaf_frame.cuh"
#include "scan.cuh"

namespace cspt {

uint64_t& last_fallbacks()
{
  static thread_local uint64_t n = 0;
  return n;
}
uint64_t& last_group_scans()
{
  static thread_local uint64_t n = 0;
  return n;
}
uint64_t& last_f64_segments()
{
  static thread_local uint64_t n = 0;
  return n;
}

namespace {

template <typename T>
__device__ inline T dot_fma(T ax, T ay, T bx, T by)
{
  return fma_rn(ax, bx, ay * by);
}

// (the quotient r is only formed where the result depends on it: when
// d3 <= 0 the reference's expression yields fmin(d0, d1) whatever r is)
template <typename T>
__device__ inline T segment_dist2(T px, T py, T ax, T ay, T bx, T by)
{
  T const v1x = px - ax, v1y = py - ay;
  T const v2x = px - bx, v2y = py - by;
  T const d0  = dot_fma(v1x, v1y, v1x, v1y);
  T const d1  = dot_fma(v2x, v2y, v2x, v2y);
  T const ex = bx - ax, ey = by - ay;
  T const d3  = dot_fma(px - ax, py - ay, ex, ey);
  if (d3 <= T{0}) return fmin(d0, d1);
  T const d2 = dot_fma(ex, ey, ex, ey);
  T const r  = d3 * d3 / d2;
  return r >= d2 ? fmin(d0, d1) : d0 - r;
}

// quadtree_point_to_nearest_linestring.cuh:279-294 — lhs is the running
// value, rhs the next candidate.
template <typename T>
__device__ inline bool take_rhs(T dl, uint32_t il, T dr, uint32_t ir)
{
  if (dl == T{0}) return true;
  if (dr == T{0}) return false;
  if (dl == dr) return !(il < ir);
  return !(dl < dr);
}

__global__ void init_rows_kernel(size_t n, uint32_t* __restrict__ opt, uint32_t* __restrict__ ols,
                                 void* __restrict__ od, int dsize)
{
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    opt[i] = static_cast<uint32_t>(i);
    ols[i] = 0xFFFFFFFFu;
    if (dsize == 8)
      static_cast<double*>(od)[i] = 0.0;
    else
      static_cast<float*>(od)[i] = 0.0f;
  }
}

constexpr int kSegChunk = 8;  // segments per pruning box

// Bounding boxes (minx, miny, maxx, maxy) of the linestrings and of their
// chunks of kSegChunk segments, in float32 rounded outward; a box with a
// non-finite coordinate is the whole plane.  Chunk c of linestring l is at
// v0 / kSegChunk + l + c (v0 its first vertex): the ranges of successive
// linestrings do not overlap, and no scan is needed to place them.
struct LsBounds {
  float4 const* ls;  // null: nothing is pruned (a call short of memory)
  float4 const* chunk;
  uint32_t slots;  // chunk boxes; offsets that leave them are not pruned by chunk
  float2 const* vertex;  // the vertices to nearest float32 (exact method)
  uint32_t nv;           // how many; offsets beyond are not pruned by segment
};
__host__ __device__ inline size_t chunk_slots(size_t nv, size_t nls)
{
  return nv / kSegChunk + nls + 1;
}

__device__ inline float float_down(double v) { return __double2float_rd(v); }
__device__ inline float float_up(double v) { return __double2float_ru(v); }
__device__ inline float float_down(float v) { return v; }
__device__ inline float float_up(float v) { return v; }

struct BoundBox {
  float4 b;  // empty: (inf, inf, -inf, -inf)
  __device__ BoundBox() : b(make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY)) {}
  template <typename T>
  __device__ void add(T x, T y)
  {
    if (isfinite(x) && isfinite(y)) {
      b.x = fminf(b.x, float_down(x));
      b.y = fminf(b.y, float_down(y));
      b.z = fmaxf(b.z, float_up(x));
      b.w = fmaxf(b.w, float_up(y));
    } else {
      b = make_float4(-INFINITY, -INFINITY, INFINITY, INFINITY);
    }
  }
  __device__ void add(float4 o)
  {
    b = make_float4(fminf(b.x, o.x), fminf(b.y, o.y), fmaxf(b.z, o.z), fmaxf(b.w, o.w));
  }
};

// One warp per linestring, a lane per chunk.
template <typename T>
__global__ void __launch_bounds__(256)
  ls_bounds_kernel(uint32_t const* __restrict__ lso, size_t nls, T const* __restrict__ lx,
                   T const* __restrict__ ly, size_t slots, float4* __restrict__ ls_box,
                   float4* __restrict__ chunk_box, uint32_t nv, float2* __restrict__ vertex)
{
  int const lane      = threadIdx.x & 31;
  size_t const nwarps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  for (size_t l = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5; l < nls;
       l += nwarps) {
    uint32_t const v0   = lso[l], v1 = lso[l + 1];
    uint32_t const nseg = v1 > v0 + 1 ? v1 - v0 - 1 : 0;
    size_t const base   = v0 / kSegChunk + l;
    BoundBox all;
    for (uint32_t c = lane; c * kSegChunk < nseg; c += 32) {
      BoundBox box;
      uint32_t const s0 = v0 + c * kSegChunk, s1 = min(s0 + kSegChunk, v0 + nseg);
      for (uint32_t v = s0; v <= s1; ++v) {
        T const x = lx[v], y = ly[v];
        box.add(x, y);
        if ((v < s1 || v + 1 == v1) && v < nv)
          vertex[v] = make_float2(static_cast<float>(x), static_cast<float>(y));
      }
      if (base + c < slots) chunk_box[base + c] = box.b;
      all.add(box.b);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      all.add(make_float4(__shfl_xor_sync(0xFFFFFFFFu, all.b.x, o),
                          __shfl_xor_sync(0xFFFFFFFFu, all.b.y, o),
                          __shfl_xor_sync(0xFFFFFFFFu, all.b.z, o),
                          __shfl_xor_sync(0xFFFFFFFFu, all.b.w, o)));
    if (lane == 0) ls_box[l] = all.b;
  }
}

// A lower bound of the squared segment distance that the reference's
// expression gives in type T, for every segment with both ends in box b and a
// finite point in [xl, xu] x [yl, yu].  The distance to the box is rounded
// down throughout.  With u the type's unit roundoff (2^-53, 2^-24), D^2 the
// largest squared distance to the box and v, e the expression's vectors, its
// value is within 21 u D^2 of the exact one: 4 u |v|^2 for d0, 5 u |v| |e| for
// d3 and 4 u |e|^2 for d2, hence 16 u |v|^2 for r = d3^2 / d2, and u for the
// difference; underflow adds less than 2^-120.  The bound takes 32 u D^2.
struct PointBounds {
  float xl, xu, yl, yu;
  bool finite;
};
template <typename T>
__device__ inline PointBounds point_bounds(T x, T y)
{
  return PointBounds{float_down(x), float_up(x), float_down(y), float_up(y),
                     isfinite(x) && isfinite(y)};
}
template <typename T>
__device__ inline float box_lower(PointBounds const& p, float4 b)
{
  constexpr float k32u = sizeof(T) == 8 ? 3.5527136788005009e-15f : 1.9073486328125e-06f;
  float const dx = fmaxf(fmaxf(__fsub_rd(b.x, p.xu), __fsub_rd(p.xl, b.z)), 0.0f);
  float const dy = fmaxf(fmaxf(__fsub_rd(b.y, p.yu), __fsub_rd(p.yl, b.w)), 0.0f);
  float const fx = fmaxf(__fsub_ru(p.xu, b.x), __fsub_ru(b.z, p.xl));
  float const fy = fmaxf(__fsub_ru(p.yu, b.y), __fsub_ru(b.w, p.yl));
  float const lb = __fadd_rd(__fmul_rd(dx, dx), __fmul_rd(dy, dy));
  float const D2 = __fadd_ru(__fmul_ru(fx, fx), __fmul_ru(fy, fy));
  return __fsub_rd(lb, __fmaf_ru(D2, k32u, 7.52316384526264e-37f));
}

template <typename T>
__device__ inline float linestring_lower(PointBounds const& p, LsBounds const& b, uint32_t l)
{
  return b.ls ? box_lower<T>(p, b.ls[l]) : -INFINITY;
}

// An upper bound of the squared distance that the reference's expression gives
// for a segment that starts at a vertex known to nearest float32, where it gives a
// number: at most |p - v|^2 (its d0), the coordinates off by 2^-24 of their
// magnitude and the roundings of d0 and of this by less than 2^-20.  Infinite where
// v or the point is not finite.  Where the segment's other end is not finite, or its
// squares overflow or underflow, the expression is not a number and the segment
// gives no distance at all: whoever uses the bound asks holds_bound afterwards.
__device__ inline float vertex_upper(PointBounds const& p, float2 v)
{
  float const dx = fmaxf(__fsub_ru(p.xu, v.x), __fsub_ru(v.x, p.xl));
  float const dy = fmaxf(__fsub_ru(p.yu, v.y), __fsub_ru(v.y, p.yl));
  float const ex = __fmaf_ru(fabsf(v.x), 1.1920928955078125e-07f, dx);  // 2^-23
  float const ey = __fmaf_ru(fabsf(v.y), 1.1920928955078125e-07f, dy);
  float const u  = __fmul_ru(__fadd_ru(__fmul_ru(ex, ex), __fmul_ru(ey, ey)), 1.000002f);
  return u < INFINITY ? __fadd_ru(u, 1.0e-37f) : INFINITY;
}

// box_lower of a segment between two such vertices (not finite: a bound below
// everything).
template <typename T>
__device__ inline float segment_lower(PointBounds const& p, float2 a, float2 b)
{
  float const ex = 1.1920928955078125e-07f * fmaxf(fabsf(a.x), fabsf(b.x));
  float const ey = 1.1920928955078125e-07f * fmaxf(fabsf(a.y), fabsf(b.y));
  if (!(ex < INFINITY && ey < INFINITY)) return -INFINITY;
  return box_lower<T>(p, make_float4(__fsub_rd(fminf(a.x, b.x), ex), __fsub_rd(fminf(a.y, b.y), ey),
                                     __fadd_ru(fmaxf(a.x, b.x), ex),
                                     __fadd_ru(fmaxf(a.y, b.y), ey)));
}

// The running winner of the reference's fold, and the squared distance (in
// float32, rounded up) beyond which a candidate's root is larger than the
// winner's: such a candidate is not zero and never taken.  Nothing is passed
// over while there is no winner, its distance is zero (it yields to the next
// candidate whatever that is) or not a number.
template <typename T>
struct Fold {
  bool have    = false;
  uint32_t bid = 0;
  T bd         = 0;
  float far    = INFINITY;

  __device__ void take(T d, uint32_t lid)
  {
    if (!have || take_rhs<T>(bd, bid, d, lid)) {
      bid = lid;
      bd  = d;
      // (1 + 2^-20) covers the roundings of the root and of the square
      far = bd > T{0} ? __fmul_ru(__fmul_ru(float_up(bd), float_up(bd)), 1.0000009536743164f)
                      : INFINITY;
    }
    have = true;
  }
};

// Whether a fold that passed over what lies beyond `bound` is the whole fold's:
// every linestring it took is at a positive distance, and its winner lies within
// the bound, so what was passed over is beyond the winner.  (A fold of no
// candidates holds too.)  The bound is above the square of any distance that it
// comes from by 2^-19, so its own linestring passes.
template <typename T>
__device__ inline bool holds_bound(Fold<T> const& f, bool zero, float bound)
{
  if (bound == INFINITY || !f.have) return true;
  return !zero && __fmul_rd(float_down(f.bd), float_down(f.bd)) < bound;
}

// point_linestring_distance.cuh:32-51 without the chunks and segments that
// cannot change the fold: those beyond `far`, and those beyond the smallest
// distance so far.
template <typename T>
__device__ inline T linestring_distance(T px, T py, PointBounds const& pb, T const* lx,
                                        T const* ly, uint32_t v0, uint32_t v1,
                                        LsBounds const& bounds, uint32_t slot, float far)
{
  T ds                = std::numeric_limits<T>::max();
  uint32_t const nseg = v1 > v0 + 1 ? v1 - v0 - 1 : 0;
  for (uint32_t c = 0; c * kSegChunk < nseg; ++c) {
    if (pb.finite && slot + c < bounds.slots && box_lower<T>(pb, bounds.chunk[slot + c]) > far)
      continue;
    uint32_t const s0 = v0 + c * kSegChunk, s1 = min(s0 + kSegChunk, v0 + nseg);
    bool const cull = pb.finite && s1 < bounds.nv;
    float2 fa       = cull ? bounds.vertex[s0] : make_float2(0.0f, 0.0f);
    for (uint32_t s = s0; s < s1; ++s) {
      if (cull) {
        float2 const fb = bounds.vertex[s + 1];
        bool const out  = segment_lower<T>(pb, fa, fb) > far;
        fa              = fb;
        if (out) continue;
      }
      ds  = fmin(ds, segment_dist2<T>(px, py, lx[s], ly[s], lx[s + 1], ly[s + 1]));
      far = fminf(far, float_up(ds));
    }
  }
  return sqrt(ds);
}

// Up to this many points take a warp each (exact method, and the groups the
// filtered kernel leaves).  Whole calls, a warp per point against a lane: 1081
// points x 3190 linestrings 585 and 1234 us, 2000 x 20k 4.7 and 19.4 ms, 1620 x 72
// 459 and 541 us; 5000 x 1000 1081 to 1422 and 998 to 1067 us, 20k x 301 2003 and
// 715 us.  What the filtered kernel leaves counts by its own points: 1M points x 3000
// linestrings with 2000 (8000) more about one leaf 1230 us (1871), by the points of
// the whole call 2299 (5683).
constexpr size_t kWarpPoints = 4096;
// warps that share a group: a warp per point, a lane per point
constexpr uint32_t kPointSplit = 64, kLaneSplit = 8;

// Whether the groups that the filtered kernel left are this kernel's: both kernels
// are launched and the number of their points decides (count: [0] the groups,
// [1] their points).
template <bool Few>
__device__ inline bool takes_left(uint32_t const* groups, uint32_t const* count)
{
  return !groups || (count[1] <= kWarpPoints) == Few;
}

// A lane per point; the candidates of its group in pair order.  `split` warps
// share a group.  `groups`: those that the filtered kernel left (which may have
// left its bound in place of the distance), or all where it is null.  Bound by the float64 pipe (two lanes a cycle and SM) and, on
// few points, by one warp's chain of candidates, hence the split.  20k points,
// 301 linestrings of 2 to 64 segments: the kernel took 6960 us with every
// candidate evaluated, 595 us with the boxes of linestrings and chunks, 280 us
// with those of segments and the bound from the chunks' first vertices (the call
// 7652, 881 and 572 us).
template <typename T>
__global__ void __launch_bounds__(256)
  nearest_kernel(uint32_t const* __restrict__ groups, uint32_t const* __restrict__ count,
                 uint32_t const* __restrict__ group_start, uint32_t const* __restrict__ ngroups_p,
                 size_t npairs, uint32_t split, uint32_t const* __restrict__ pair_ls,
                 uint32_t const* __restrict__ pair_quad, uint32_t const* __restrict__ qlen,
                 uint32_t const* __restrict__ qoff, PointSource<T> const src, size_t npi,
                 uint32_t const* __restrict__ lso, size_t nls, T const* __restrict__ lx,
                 T const* __restrict__ ly, LsBounds const bounds, uint32_t* __restrict__ opt,
                 uint32_t* __restrict__ ols, T* __restrict__ od)
{
  if (!takes_left<false>(groups, count)) return;
  int const lane       = threadIdx.x & 31;
  size_t const warps   = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  size_t const ngroups = *ngroups_p, n = *count;
  for (size_t t = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5;
       t < n * split; t += warps) {
    // (all groups' first parts, then their second parts: leaves with few points
    // have no later ones, and every warp must get its share of the first)
    size_t const part = t / n, i = t - part * n;
    size_t const g      = groups ? groups[i] : i;
    uint32_t const k0   = group_start[g];
    uint32_t const k1   = (g + 1 < ngroups) ? group_start[g + 1] : static_cast<uint32_t>(npairs);
    uint32_t const quad = pair_quad[k0];
    uint32_t const len  = qlen[quad];
    uint64_t const off  = qoff[quad];
    for (uint32_t c = static_cast<uint32_t>(part) * 32 + lane; c < len; c += 32 * split) {
      uint64_t const pos = off + c;
      if (pos >= npi) continue;
      T px, py;
      src.load(pos, px, py);
      PointBounds const pb = point_bounds<T>(px, py);
      // No candidate beyond the distance to some chunk's first vertex can win,
      // unless that vertex's linestring turns out at distance zero (or not a
      // number), which the fold passes over, or the vertex's segment gives no
      // distance: then the point is folded again without the bound.
      float bound = INFINITY;
      for (uint32_t k = k0; k < k1 && pb.finite; ++k) {
        uint32_t const lid = pair_ls[k];
        if (lid >= nls || linestring_lower<T>(pb, bounds, lid) > bound) continue;
        uint32_t const v0 = lso[lid], v1 = lso[lid + 1];
        for (uint32_t v = v0; v + 1 < v1 && v < bounds.nv; v += kSegChunk)
          bound = fminf(bound, vertex_upper(pb, bounds.vertex[v]));
      }
      Fold<T> f;
      for (;;) {
        f         = Fold<T>{};
        f.far     = bound;
        bool zero = false;
        for (uint32_t k = k0; k < k1; ++k) {
          uint32_t const lid = pair_ls[k];
          if (lid >= nls) continue;
          if (pb.finite && linestring_lower<T>(pb, bounds, lid) > f.far) continue;
          uint32_t const v0 = lso[lid];
          T const d = linestring_distance<T>(px, py, pb, lx, ly, v0, lso[lid + 1], bounds,
                                             v0 / kSegChunk + lid, f.far);
          f.take(d, lid);
          f.far = fminf(f.far, bound);
          zero |= !(d > T{0});
        }
        if (holds_bound(f, zero, bound)) break;
        bound = INFINITY;
      }
      if (f.have) {
        opt[pos] = static_cast<uint32_t>(pos);
        ols[pos] = f.bid;
      }
      if (f.have || groups) od[pos] = f.have ? f.bd : T{0};
    }
  }
}

// The reference's fold over every candidate of a group for one point, by the
// whole warp: a lane per linestring tests its box, and those that may matter
// are taken in pair order, a lane per segment.  (By one lane over every
// segment, one point at distance zero among 5M cost 50 to 110 ms.)
template <typename T>
struct FoldArgs {
  uint32_t const* pair_ls;
  uint32_t const* lso;
  size_t nls;
  T const* lx;
  T const* ly;
  LsBounds bounds;
};

template <typename T>
__device__ void fold_warp(FoldArgs<T> const& a, uint32_t k0, uint32_t k1, T px, T py,
                          bool use_bound, Fold<T>& f)
{
  constexpr unsigned kAll = 0xFFFFFFFFu;
  int const lane          = threadIdx.x & 31;
  PointBounds const pb    = point_bounds<T>(px, py);
  // the bound of nearest_kernel, from the chunks' first vertices
  float bound = INFINITY;
  for (uint32_t kb = k0; kb < k1 && use_bound && pb.finite; kb += 32) {
    uint32_t const k   = kb + static_cast<uint32_t>(lane);
    uint32_t const lid = k < k1 ? a.pair_ls[k] : 0xFFFFFFFFu;
    if (k < k1 && lid < a.nls && !(linestring_lower<T>(pb, a.bounds, lid) > bound)) {
      uint32_t const v1 = a.lso[lid + 1];
      for (uint32_t v = a.lso[lid]; v + 1 < v1 && v < a.bounds.nv; v += kSegChunk)
        bound = fminf(bound, vertex_upper(pb, a.bounds.vertex[v]));
    }
    // (not negative: ordered as integers)
    bound = __uint_as_float(__reduce_min_sync(kAll, __float_as_uint(bound)));
  }
  for (;;) {
    f         = Fold<T>{};
    f.far     = bound;
    bool zero = false;
    for (uint32_t kb = k0; kb < k1; kb += 32) {
      uint32_t const k   = kb + static_cast<uint32_t>(lane);
      uint32_t const lid = k < k1 ? a.pair_ls[k] : 0xFFFFFFFFu;
      bool const valid   = k < k1 && lid < a.nls;
      float const lb     = valid && pb.finite ? linestring_lower<T>(pb, a.bounds, lid) : -INFINITY;
      unsigned left      = __ballot_sync(kAll, valid);
      for (;;) {
        // the next in order that is not beyond the winner so far (which a zero
        // distance or one that is not a number may give up again, so those
        // beyond it are only passed over up to here)
        unsigned const near = left & __ballot_sync(kAll, !(lb > f.far));
        if (!near) break;
        int const src = __ffs(near) - 1;
        left &= ~((2u << src) - 1u);
        uint32_t const l    = __shfl_sync(kAll, lid, src);
        uint32_t const v0   = a.lso[l], v1 = a.lso[l + 1];
        uint32_t const nseg = v1 > v0 + 1 ? v1 - v0 - 1 : 0;
        uint32_t const slot = v0 / kSegChunk + l;
        T ds                = std::numeric_limits<T>::max();
        for (uint32_t s = lane; s < nseg; s += 32) {
          uint32_t const c = slot + s / kSegChunk, v = v0 + s;
          if (pb.finite && c < a.bounds.slots && box_lower<T>(pb, a.bounds.chunk[c]) > f.far)
            continue;
          if (pb.finite && v + 1 < a.bounds.nv &&
              segment_lower<T>(pb, a.bounds.vertex[v], a.bounds.vertex[v + 1]) > f.far)
            continue;
          ds = fmin(ds, segment_dist2<T>(px, py, a.lx[v], a.ly[v], a.lx[v + 1], a.ly[v + 1]));
        }
        for (int o = 16; o > 0; o >>= 1) ds = fmin(ds, __shfl_xor_sync(kAll, ds, o));
        T const d = sqrt(ds);
        f.take(d, l);
        f.far = fminf(f.far, bound);
        zero |= !(d > T{0});
      }
    }
    if (holds_bound(f, zero, bound)) break;
    bound = INFINITY;
  }
}

// nearest_kernel with a warp per point, for few points, whose lanes would leave
// the GPU idle.
template <typename T>
__global__ void __launch_bounds__(256)
  nearest_point_kernel(uint32_t const* __restrict__ groups, uint32_t const* __restrict__ count,
                       uint32_t const* __restrict__ group_start,
                       uint32_t const* __restrict__ ngroups_p, size_t npairs, uint32_t split,
                       uint32_t const* __restrict__ pair_quad, uint32_t const* __restrict__ qlen,
                       uint32_t const* __restrict__ qoff, PointSource<T> const src, size_t npi,
                       FoldArgs<T> const a, uint32_t* __restrict__ opt,
                       uint32_t* __restrict__ ols, T* __restrict__ od)
{
  if (!takes_left<true>(groups, count)) return;
  int const lane       = threadIdx.x & 31;
  size_t const warps   = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  size_t const ngroups = *ngroups_p, n = *count;
  for (size_t t = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5;
       t < n * split; t += warps) {
    // (all groups' first parts, then their second parts: leaves with few points
    // have no later ones, and every warp must get its share of the first)
    size_t const part = t / n, i = t - part * n;
    size_t const g      = groups ? groups[i] : i;
    uint32_t const k0   = group_start[g];
    uint32_t const k1   = g + 1 < ngroups ? group_start[g + 1] : static_cast<uint32_t>(npairs);
    uint32_t const quad = pair_quad[k0];
    uint32_t const len  = qlen[quad];
    uint64_t const off  = qoff[quad];
    for (uint32_t c = static_cast<uint32_t>(part); c < len; c += split) {
      uint64_t const pos = off + c;
      if (pos >= npi) break;
      T px, py;
      src.load(pos, px, py);
      Fold<T> f;
      fold_warp<T>(a, k0, k1, px, py, true, f);
      if (lane == 0) {
        if (f.have) {
          opt[pos] = static_cast<uint32_t>(pos);
          ols[pos] = f.bid;
        }
        // (the filtered kernel may have left its bound here)
        od[pos] = f.have ? f.bd : T{0};
      }
    }
  }
}

// ---------------------------------------------------------------------------
// float32 filter (float64 inputs)
// ---------------------------------------------------------------------------
constexpr int kSegSuper = 64;  // segments per coarse pruning box (8 chunks)
// (the coarse boxes' slots, as chunk_slots: box c of linestring l is at
// v0 / kSegSuper + l + c)
inline size_t super_slots(size_t nv, size_t nls) { return nv / kSegSuper + nls + 1; }

// Per linestring, what the segment listing needs in one 64-byte record.
struct __align__(16) LsRec {
  long long aix, aiy;  // anchor in grid steps
  float4 box;          // box of its float32 segments, anchor frame
  float maxoff;        // largest |float32 offset|
  uint32_t v0, nseg;   // first vertex, segments
  uint32_t cb;         // first chunk's slot
  uint32_t sb;         // first coarse box's slot
  uint32_t exact;      // non-finite coordinates: exact path only
  uint32_t pad[2];
};
static_assert(sizeof(LsRec) == 64, "one 64-byte record per linestring");

struct LinestringIndexView {
  long long const* aix;  // anchors in grid steps
  long long const* aiy;
  float const* maxoff;   // largest |float32 offset| of the linestring
  float4 const* chunk_box;  // (minx, miny, maxx, maxy) of 8 segments, anchor frame
  float4 const* super_box;  // the same of 64 segments
  float4 const* seg32;      // per segment start vertex: (ax, ay, bx, by), anchor frame
  uint8_t const* exact;     // non-finite coordinates: exact path only
  LsRec const* rec;
};

// per linestring: box, anchor, float32 segments, chunk boxes (one warp each)
__global__ void __launch_bounds__(256)
  ls_box_kernel(uint32_t const* __restrict__ lso, size_t nls, double const* __restrict__ lx,
                double const* __restrict__ ly, double4_16a* __restrict__ box, uint8_t* exact)
{
  int const lane      = threadIdx.x & 31;
  size_t const nwarps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  for (size_t l = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5; l < nls;
       l += nwarps) {
    uint32_t const v0 = lso[l], v1 = lso[l + 1];
    double mnx = INFINITY, mny = INFINITY, mxx = -INFINITY, mxy = -INFINITY;
    bool bad = false;
    for (uint32_t v = v0 + lane; v < v1; v += 32) {
      double const x = lx[v], y = ly[v];
      bad |= !(isfinite(x) && isfinite(y));
      mnx = fmin(mnx, x);
      mny = fmin(mny, y);
      mxx = fmax(mxx, x);
      mxy = fmax(mxy, y);
    }
    for (int o = 16; o > 0; o >>= 1) {
      mnx = fmin(mnx, __shfl_xor_sync(0xFFFFFFFFu, mnx, o));
      mny = fmin(mny, __shfl_xor_sync(0xFFFFFFFFu, mny, o));
      mxx = fmax(mxx, __shfl_xor_sync(0xFFFFFFFFu, mxx, o));
      mxy = fmax(mxy, __shfl_xor_sync(0xFFFFFFFFu, mxy, o));
    }
    bad = __any_sync(0xFFFFFFFFu, bad);
    if (lane == 0) {
      box[l]         = make_double4_16a(mnx, mny, mxx, mxy);
      exact[l]       = bad ? 1 : 0;
    }
  }
}

__global__ void __launch_bounds__(1024) ls_grid_kernel(double4_16a const* __restrict__ box, size_t nls,
                                                       double* grid)
{
  __shared__ double part[32];
  double m = 0;
  for (size_t l = threadIdx.x; l < nls; l += blockDim.x) {
    double4_16a const b = box[l];
    double const v[4] = {b.x, b.y, b.z, b.w};
    for (double a : v)
      if (isfinite(a)) m = fmax(m, fabs(a));
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = part[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if (threadIdx.x == 0) {
      int e = 0;
      frexp(m > 0.0 ? m : 1.0, &e);
      *grid = ldexp(1.0, e - 22);
    }
  }
}

__global__ void __launch_bounds__(256)
  ls_fill_kernel(uint32_t const* __restrict__ lso, size_t nls, double const* __restrict__ lx,
                 double const* __restrict__ ly, double4_16a const* __restrict__ box,
                 double const* __restrict__ gridp, uint8_t const* __restrict__ exact,
                 long long* aix, long long* aiy, float* maxoff, float4* chunk_box, float4* seg32,
                 LsRec* rec, size_t slots, float4* __restrict__ abs_ls,
                 float4* __restrict__ abs_chunk, size_t sslots, float4* __restrict__ super_box,
                 uint32_t nv, float2* __restrict__ vertex)
{
  int const lane      = threadIdx.x & 31;
  size_t const nwarps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  double const g      = *gridp;
  for (size_t l = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5; l < nls;
       l += nwarps) {
    uint32_t const v0 = lso[l], v1 = lso[l + 1];
    double4_16a const b   = box[l];
    double rx = v1 > v0 ? rint((b.x + b.z) * 0.5 / g) : 0.0;
    double ry = v1 > v0 ? rint((b.y + b.w) * 0.5 / g) : 0.0;
    if (!(fabs(rx) < 4.0e18)) rx = 0.0;
    if (!(fabs(ry) < 4.0e18)) ry = 0.0;
    double const cx = rx * g, cy = ry * g;
    uint32_t const nseg = v1 > v0 + 1 ? v1 - v0 - 1 : 0;
    uint32_t const nch  = (nseg + kSegChunk - 1) / kSegChunk;
    uint32_t const cb   = v0 / kSegChunk + static_cast<uint32_t>(l);
    float m             = 0.0f;
    float4 lbx          = make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY);
    BoundBox all;  // the boxes of LsBounds, for points folded over every candidate
    // lane per chunk, eight lanes per coarse box
    uint32_t const sb = v0 / kSegSuper + static_cast<uint32_t>(l);
    for (uint32_t c0 = 0; c0 < nch; c0 += 32) {
      uint32_t const c = c0 + static_cast<uint32_t>(lane);
      float4 cbx = make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY);
      if (c < nch) {
        uint32_t const s0 = v0 + c * kSegChunk;
        uint32_t const s1 = min(s0 + kSegChunk, v0 + nseg);
        BoundBox abs_box;
        abs_box.add(lx[s0], ly[s0]);
        for (uint32_t sg = s0; sg < s1; ++sg) {
          abs_box.add(lx[sg + 1], ly[sg + 1]);
          if (sg < nv)
            vertex[sg] = make_float2(static_cast<float>(lx[sg]), static_cast<float>(ly[sg]));
          if (sg + 2 == v1 && sg + 1 < nv)
            vertex[sg + 1] =
              make_float2(static_cast<float>(lx[sg + 1]), static_cast<float>(ly[sg + 1]));
          float4 e;
          e.x       = static_cast<float>(lx[sg] - cx);
          e.y       = static_cast<float>(ly[sg] - cy);
          e.z       = static_cast<float>(lx[sg + 1] - cx);
          e.w       = static_cast<float>(ly[sg + 1] - cy);
          seg32[sg] = e;
          cbx.x     = fminf(cbx.x, fminf(e.x, e.z));
          cbx.y     = fminf(cbx.y, fminf(e.y, e.w));
          cbx.z     = fmaxf(cbx.z, fmaxf(e.x, e.z));
          cbx.w     = fmaxf(cbx.w, fmaxf(e.y, e.w));
          m = fmaxf(m, fmaxf(fmaxf(fabsf(e.x), fabsf(e.y)), fmaxf(fabsf(e.z), fabsf(e.w))));
        }
        all.add(abs_box.b);
        if (cb + c < slots) {
          chunk_box[cb + c] = cbx;
          if (abs_chunk) abs_chunk[cb + c] = abs_box.b;
        }
      }
      float4 sbx = cbx;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1)
        sbx = make_float4(fminf(sbx.x, __shfl_xor_sync(0xFFFFFFFFu, sbx.x, o)),
                          fminf(sbx.y, __shfl_xor_sync(0xFFFFFFFFu, sbx.y, o)),
                          fmaxf(sbx.z, __shfl_xor_sync(0xFFFFFFFFu, sbx.z, o)),
                          fmaxf(sbx.w, __shfl_xor_sync(0xFFFFFFFFu, sbx.w, o)));
      if (c < nch && (lane & 7) == 0 && sb + (c >> 3) < sslots) super_box[sb + (c >> 3)] = sbx;
      lbx = make_float4(fminf(lbx.x, cbx.x), fminf(lbx.y, cbx.y), fmaxf(lbx.z, cbx.z),
                        fmaxf(lbx.w, cbx.w));
    }
    m     = warp_max(m);
    lbx.x = warp_min(lbx.x);
    lbx.y = warp_min(lbx.y);
    lbx.z = warp_max(lbx.z);
    lbx.w = warp_max(lbx.w);
    all.b = make_float4(warp_min(all.b.x), warp_min(all.b.y), warp_max(all.b.z),
                        warp_max(all.b.w));
    if (lane == 0) {
      if (abs_ls) abs_ls[l] = all.b;
      aix[l]    = static_cast<long long>(rx);
      aiy[l]    = static_cast<long long>(ry);
      maxoff[l] = m;
      LsRec r{};
      r.aix    = static_cast<long long>(rx);
      r.aiy    = static_cast<long long>(ry);
      r.box    = lbx;
      r.maxoff = m;
      r.v0     = v0;
      r.nseg   = nseg;
      r.cb     = cb;
      r.sb     = sb;
      r.exact  = exact[l];
      rec[l]   = r;
    }
  }
}

// float32 estimate of the reference's squared segment distance and a bound on
// |estimate - float64 value|.  With d = 2 u32 M bounding each coordinate's
// mapping error (point in the leaf frame, segment in the linestring frame,
// M the largest offset), s = |v1|, t = |e|:
//   d0, d1: 4 d s + 4 u32 s^2 (and with w = |v2| <= s + t),
//   d2: 4 d t + 4 u32 t^2, d3: 2 d (s + t) + 4 u32 s t,
//   d0 - d3^2/d2 adds r (dd3/d3 * 2 + dd2/d2), i.e. up to 4 d s^2 / t;
// the branch choice near a projection end changes the value by the square
// of those errors only (the two branches meet there).  1/t comes from the
// approximate reciprocal square root (2^-22.9) and s from the approximate square
// root: r = d3^2 (1/t)^2 is off by 6 u32 s^2 more.  The bound below takes more
// than twice the sum of all that plus 2^-40 of the magnitudes for the float64
// rounding; t -> 0 makes it infinite, which sends the segment to float64.
__device__ inline void seg_estimate(float qx, float qy, float4 e, float dm, float& est,
                                    float& err)
{
  float const v1x = qx - e.x, v1y = qy - e.y;
  float const v2x = qx - e.z, v2y = qy - e.w;
  float const ex = e.z - e.x, ey = e.w - e.y;
  float const d0 = __fmaf_rn(v1x, v1x, v1y * v1y);
  float const d1 = __fmaf_rn(v2x, v2x, v2y * v2y);
  float const d2 = __fmaf_rn(ex, ex, ey * ey);
  float const d3 = __fmaf_rn(v1x, ex, v1y * ey);
  float it, sv;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(it) : "f"(d2));
  asm("sqrt.approx.f32 %0, %1;" : "=f"(sv) : "f"(d0));
  float const q  = d3 * it;
  float const r  = q * q;
  est            = (d3 <= 0.0f || r >= d2) ? fminf(d0, d1) : d0 - r;
  float const tv = d2 * it;
  float const u32 = 5.960464477539063e-08f;
  err = 4.0f * (dm * (8.0f * sv + 4.0f * tv + 4.0f * d0 * it) +
                u32 * (12.0f * d0 + 8.0f * sv * tv + 4.0f * d2)) +
        9.094947017729282e-13f * (d0 + d2) + 7.52316384526264e-37f;
  if (!(err < INFINITY)) err = INFINITY;
}

// squared distance from q to a box widened by tol, shrunk by 2^-30 relative
__device__ inline float box_lb(float qx, float qy, float4 b, float tol)
{
  float const dx = fmaxf(fmaxf(b.x - tol - qx, 0.0f), qx - b.z - tol);
  float const dy = fmaxf(fmaxf(b.y - tol - qy, 0.0f), qy - b.w - tol);
  return __fmaf_rn(dx, dx, dy * dy) * 0.9999999990686774f;
}

// squared distance between two boxes, each side widened by tol, shrunk by
// 2^-30 relative: a lower bound of box_lb for every point of box a
__device__ inline float boxbox_lb(float4 a, float4 b, float tol)
{
  float const dx = fmaxf(fmaxf(b.x - tol - a.z, 0.0f), a.x - b.z - tol);
  float const dy = fmaxf(fmaxf(b.y - tol - a.w, 0.0f), a.y - b.w - tol);
  return __fmaf_rn(dx, dx, dy * dy) * 0.9999999990686774f;
}

// Arguments of the filtered nearest-linestring kernel.
struct NearestArgs {
  uint32_t const* group_start;
  uint32_t const* ngroups_p;
  size_t npairs;
  uint32_t const* pair_ls;
  uint32_t const* pair_quad;
  uint32_t const* qlen;
  uint32_t const* qoff;
  PointSource<double> src;
  size_t npi;
  uint32_t const* lso;
  size_t nls;
  double const* lx;
  double const* ly;
  float2 const* u;
  LeafFrame const* frames;
  LinestringIndexView li;
  LsBounds bounds;
  float gf;
  uint32_t* opt;
  uint32_t* ols;
  double* od;
  unsigned long long* stats;  // [0] points folded over every candidate, [1] groups scanned whole
  unsigned long long* next_group;
  uint32_t* left;   // groups that the listing cannot take
  uint32_t* nleft;  // [0] how many, [1] their points
};

// Folds the points of the lanes that ask for it, one after the other.
__device__ inline void fold_lanes(NearestArgs const& a, uint32_t k0, uint32_t k1, bool ask,
                                  double px, double py, bool& have, uint32_t& bid, double& bd,
                                  uint32_t& nfb)
{
  for (unsigned m = __ballot_sync(0xFFFFFFFFu, ask); m; m &= m - 1u) {
    int const src = __ffs(m) - 1;
    Fold<double> f;
    // (mostly points at a zero distance, which would drop the bound again)
    fold_warp<double>(FoldArgs<double>{a.pair_ls, a.lso, a.nls, a.lx, a.ly, a.bounds}, k0, k1,
                      __shfl_sync(0xFFFFFFFFu, px, src), __shfl_sync(0xFFFFFFFFu, py, src), false,
                      f);
    if (static_cast<int>(threadIdx.x & 31) == src) {
      ++nfb;
      have = f.have;
      bid  = f.bid;
      bd   = f.bd;
    }
  }
}

// The group's segment list (per warp, in shared memory): the candidate
// segments whose box lies within a radius of the leaf's point box, each in
// the leaf's float32 frame, with its global start vertex and its
// linestring, in no particular order.
constexpr int kNearWarps    = 4;    // warps per block
constexpr uint32_t kNearCap = 384;  // listed segments per warp
static_assert(kNearCap <= 65536, "candidate slots hold 16-bit list positions");
// float64 candidates per point evaluated in lockstep rounds (more are taken
// one lane at a time)
constexpr uint32_t kNearCand = 4;
struct NearList {
  float4 e[kNearCap];
  uint32_t seg[kNearCap];
  uint32_t lid[kNearCap];
};
constexpr uint32_t kListOverflow = 0xFFFFFFFEu;  // more than kNearCap segments
constexpr uint32_t kListFrame    = 0xFFFFFFFFu;  // a linestring outside the float32 frames

// Lists the segments of the group's linestrings whose box is within squared
// distance r2 of the leaf's point box (box-to-box lower bound with the
// filter's margin tol, computed in each linestring's frame; the leaf box
// maps into that frame monotonically, so it holds every point's mapped
// offset and the bound is below each point's own box_lb).  Four filters,
// each on every lane: 32 candidate linestrings at a time, each lane loading
// one linestring's 64-byte record and testing its whole box; the coarse boxes
// (64 segments) of the linestrings that pass, flattened over the lanes (a lane
// finds its box's linestring by a binary search over the lanes' running
// counts); four near coarse boxes at a time, eight lanes per box, one chunk
// each; four near chunks at a time, eight lanes per chunk, one segment each.  Listed segments are stored in the leaf frame, rounded once from the
// float64 vertices; mg receives the largest magnitude of the leaf frame (its
// points' and the listed segments' offsets), which bounds their errors.
// Returns the count, kListOverflow or kListFrame.
__device__ uint32_t list_segments(NearestArgs const& a, NearList& L, uint32_t k0, uint32_t k1,
                                  LeafFrame const& lf, float r2, float& mg)
{
  LinestringIndexView const& li = a.li;
  constexpr unsigned kAll       = 0xFFFFFFFFu;
  int const lane                = threadIdx.x & 31;
  unsigned const lt             = (1u << lane) - 1u;
  uint32_t n                    = 0;
  float m                       = lf.m;
  for (uint32_t kb = k0; kb < k1; kb += 32) {
    // this lane's linestring: its frame relative to the leaf and whether its
    // whole box is near the leaf box
    uint32_t const k = kb + static_cast<uint32_t>(lane);
    uint32_t lid     = 0;
    bool valid       = k < k1;
    if (valid) {
      lid   = a.pair_ls[k];
      valid = lid < a.nls;
    }
    LsRec r{};
    if (valid) r = li.rec[lid];
    bool bad = false;
    float4 lb{};
    float tol    = 0.0f;
    uint32_t nsb = 0;
    if (valid) {
      long long const dix = r.aix - lf.ix, diy = r.aiy - lf.iy;
      bad = r.exact || dix <= -16777216LL || dix >= 16777216LL || diy <= -16777216LL ||
            diy >= 16777216LL;
      if (!bad) {
        float const sx = static_cast<float>(static_cast<int>(dix)) * a.gf;
        float const sy = static_cast<float>(static_cast<int>(diy)) * a.gf;
        lb             = make_float4(lf.uxmin - sx, lf.uymin - sy, lf.uxmax - sx, lf.uymax - sy);
        float const mk = fmaxf(fmaxf(r.maxoff, lf.m), fmaxf(fmaxf(fabsf(lb.x), fabsf(lb.y)),
                                                            fmaxf(fabsf(lb.z), fabsf(lb.w))));
        tol            = 4.76837158203125e-07f * mk;
        if (boxbox_lb(lb, r.box, tol) <= r2) nsb = (r.nseg + kSegSuper - 1) / kSegSuper;
      }
    }
    if (__any_sync(kAll, bad)) return kListFrame;
    // running coarse box counts over the lanes
    uint32_t incl = nsb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t const t = __shfl_up_sync(kAll, incl, o);
      if (lane >= o) incl += t;
    }
    uint32_t const total = __shfl_sync(kAll, incl, 31);
    for (uint32_t c0 = 0; c0 < total; c0 += 32) {
      uint32_t const c = c0 + static_cast<uint32_t>(lane);
      // the coarse box's linestring: the first lane whose running count exceeds c
      int ow = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        uint32_t const v = __shfl_sync(kAll, incl, ow + step - 1);
        if (v <= c) ow += step;
      }
      ow = ow < 31 ? ow : 31;
      float4 const wlb    = make_float4(__shfl_sync(kAll, lb.x, ow), __shfl_sync(kAll, lb.y, ow),
                                        __shfl_sync(kAll, lb.z, ow), __shfl_sync(kAll, lb.w, ow));
      float const wtol    = __shfl_sync(kAll, tol, ow);
      uint32_t const wsb  = __shfl_sync(kAll, r.sb, ow);
      uint32_t const winc = __shfl_sync(kAll, incl, ow);
      uint32_t const wnsb = __shfl_sync(kAll, nsb, ow);
      uint32_t const sc   = c - (winc - wnsb);  // the box within its linestring
      bool const wnear    = c < total && boxbox_lb(wlb, li.super_box[wsb + sc], wtol) <= r2;
      unsigned wm         = __ballot_sync(kAll, wnear);
      while (wm) {
        // lane l expands the (l / 8)-th remaining near box, chunk l % 8; its
        // linestring is held by lane ow of that box's lane
        unsigned wl = wm;
        for (int t = 0; t < (lane >> 3); ++t) wl &= wl - 1u;
        int const wsrc       = wl ? __ffs(wl) - 1 : 0;
        int const own        = __shfl_sync(kAll, ow, wsrc);
        uint32_t const ch    = __shfl_sync(kAll, sc, wsrc) * (kSegSuper / kSegChunk) +
                               static_cast<uint32_t>(lane & 7);
        float4 const olb     = make_float4(__shfl_sync(kAll, lb.x, own), __shfl_sync(kAll, lb.y, own),
                                           __shfl_sync(kAll, lb.z, own), __shfl_sync(kAll, lb.w, own));
        float const otol     = __shfl_sync(kAll, tol, own);
        uint32_t const olid  = __shfl_sync(kAll, lid, own);
        uint32_t const ov0   = __shfl_sync(kAll, r.v0, own);
        uint32_t const onseg = __shfl_sync(kAll, r.nseg, own);
        uint32_t const ocb   = __shfl_sync(kAll, r.cb, own);
        for (int t = 0; t < 4 && wm; ++t) wm &= wm - 1u;
        bool const near = wl && ch * kSegChunk < onseg &&
                          boxbox_lb(olb, li.chunk_box[ocb + ch], otol) <= r2;
        unsigned cm     = __ballot_sync(kAll, near);
        while (cm) {
          // lane l expands the (l / 8)-th remaining near chunk, segment l % 8;
          // that chunk's linestring fields are held by lane src
          unsigned mm = cm;
          for (int t = 0; t < (lane >> 3); ++t) mm &= mm - 1u;
          int const src       = mm ? __ffs(mm) - 1 : 0;
          float4 const slb    = make_float4(__shfl_sync(kAll, olb.x, src), __shfl_sync(kAll, olb.y, src),
                                            __shfl_sync(kAll, olb.z, src), __shfl_sync(kAll, olb.w, src));
          float const stol    = __shfl_sync(kAll, otol, src);
          uint32_t const slid = __shfl_sync(kAll, olid, src);
          uint32_t const sv0  = __shfl_sync(kAll, ov0, src);
          uint32_t const snsg = __shfl_sync(kAll, onseg, src);
          uint32_t const sch  = __shfl_sync(kAll, ch, src);
          uint32_t const sg   = sv0 + sch * kSegChunk + static_cast<uint32_t>(lane & 7);
          bool keep           = false;
          if (mm && sg < sv0 + snsg) {
            float4 const e   = li.seg32[sg];
            float4 const sbx = make_float4(fminf(e.x, e.z), fminf(e.y, e.w), fmaxf(e.x, e.z),
                                           fmaxf(e.y, e.w));
            keep             = boxbox_lb(slb, sbx, stol) <= r2;
          }
          unsigned const km = __ballot_sync(kAll, keep);
          if (n + __popc(km) > kNearCap) return kListOverflow;
          if (keep) {
            // the segment in the leaf frame, rounded once from the float64
            // vertices: its error is a float32 rounding of a leaf-local value,
            // not of the linestring-frame offset (which grows with the
            // linestring's extent), so the estimates' bound stays tight
            uint32_t const slot = n + __popc(km & lt);
            float4 const el     = make_float4(static_cast<float>(a.lx[sg] - lf.ax),
                                              static_cast<float>(a.ly[sg] - lf.ay),
                                              static_cast<float>(a.lx[sg + 1] - lf.ax),
                                              static_cast<float>(a.ly[sg + 1] - lf.ay));
            L.e[slot]   = el;
            L.seg[slot] = sg;
            L.lid[slot] = slid;
            m = fmaxf(m, fmaxf(fmaxf(fabsf(el.x), fabsf(el.y)), fmaxf(fabsf(el.z), fabsf(el.w))));
          }
          n += __popc(km);
          for (int t = 0; t < 4 && cm; ++t) cm &= cm - 1u;
        }
      }
    }
  }
  __syncwarp();
  mg = warp_max(m);
  return n;
}

// An upper bound, valid for every point of the leaf, of the squared
// float64 distance to its nearest candidate segment: the smallest, over the
// candidate chunks, of the largest squared distance from the leaf box to the
// chunk's first vertex (a segment's distance is at most its start vertex's),
// each coordinate widened by the margin tol (above the mapping errors) and
// the result by 2^-20 (above the float32 rounding).  Infinite when a
// linestring lies outside the float32 frames or there is no segment.
__device__ float group_upper(NearestArgs const& a, uint32_t k0, uint32_t k1, LeafFrame const& lf)
{
  LinestringIndexView const& li = a.li;
  int const lane = threadIdx.x & 31;
  float ub       = INFINITY;
  bool frame_ok  = true;
  for (uint32_t k = k0; k < k1; ++k) {
    uint32_t const lid = a.pair_ls[k];
    if (lid >= a.nls) continue;
    long long const dix = li.aix[lid] - lf.ix, diy = li.aiy[lid] - lf.iy;
    if (li.exact[lid] || dix <= -16777216LL || dix >= 16777216LL || diy <= -16777216LL ||
        diy >= 16777216LL) {
      frame_ok = false;
      break;
    }
    float const sx  = static_cast<float>(static_cast<int>(dix)) * a.gf;
    float const sy  = static_cast<float>(static_cast<int>(diy)) * a.gf;
    float4 const lb = make_float4(lf.uxmin - sx, lf.uymin - sy, lf.uxmax - sx, lf.uymax - sy);
    float const mk  = fmaxf(fmaxf(li.maxoff[lid], lf.m),
                            fmaxf(fmaxf(fabsf(lb.x), fabsf(lb.y)), fmaxf(fabsf(lb.z), fabsf(lb.w))));
    float const tol = 4.76837158203125e-07f * mk;
    uint32_t const v0 = a.lso[lid], v1 = a.lso[lid + 1];
    uint32_t const nseg = v1 > v0 + 1 ? v1 - v0 - 1 : 0;
    for (uint32_t ch = lane; ch * kSegChunk < nseg; ch += 32) {
      float4 const e = li.seg32[v0 + ch * kSegChunk];
      float const dx = fmaxf(fabsf(e.x - lb.x), fabsf(e.x - lb.z)) + tol;
      float const dy = fmaxf(fabsf(e.y - lb.y), fabsf(e.y - lb.w)) + tol;
      ub             = fminf(ub, __fmaf_rn(dx, dx, dy * dy) * 1.0000009536743164f);
    }
  }
  ub = warp_min(ub);
  return frame_ok ? ub : INFINITY;
}

// Smallest float32 upper bound (estimate + error) of the squared distance
// from point offset (qx, qy) to the listed segments.  A segment whose box is
// farther than the running bound (box_lb, a lower bound of its distance) is
// passed over without its estimate.
__device__ inline float list_upper(NearList const& L, uint32_t n, float qx, float qy, float dm,
                                   float tol)
{
  float U = INFINITY;
  for (uint32_t t = 0; t < n; ++t) {
    float4 const e  = L.e[t];
    float4 const sb = make_float4(fminf(e.x, e.z), fminf(e.y, e.w), fmaxf(e.x, e.z),
                                  fmaxf(e.y, e.w));
    if (box_lb(qx, qy, sb, tol) > U) continue;
    float est, err;
    seg_estimate(qx, qy, e, dm, est, err);
    U = fminf(U, est + err);
  }
  return U;
}

// Whether listed segment t can reach the bound Uw from point offset
// (qx, qy): its box and then its float32 estimate (minus the estimate's
// error) are within Uw.
__device__ inline bool seg_can_reach(NearList const& L, uint32_t t, float qx, float qy, float dm,
                                     float tol, float Uw)
{
  float4 const e  = L.e[t];
  float4 const sb = make_float4(fminf(e.x, e.z), fminf(e.y, e.w), fmaxf(e.x, e.z), fmaxf(e.y, e.w));
  if (box_lb(qx, qy, sb, tol) > Uw) return false;
  float est, err;
  seg_estimate(qx, qy, e, dm, est, err);
  return !(est - err > Uw);
}

// One warp per group of pairs sharing a quadrant (handed out from a device
// counter), one lane per point.
//   1. list the segments whose box is within a radius of the leaf's point box,
//      taken from the warp's last groups (a guess: it only decides whether 3 is
//      needed; the listings are most of the kernel's instructions);
//   2. each point's float32 upper bound U over that list; r2 = the largest U
//      of the group's points: every point's nearest segment lies within r2
//      of the leaf box;
//   3. unless 1 went that far, list the segments within r2 of the leaf box: a
//      segment left out has a float64 distance above r2 >= U for every point,
//      so it can neither win nor tie;
//   4. per point: U over the list from step 2's on (one pass over the list: most
//      segments' boxes lie beyond it), then float64 (the reference's expression)
//      on every listed segment whose estimate can reach U; the winner is the
//      smallest (distance, linestring id) among them, which is the
//      reference's fold (:279-294) whenever no distance is exactly 0.  A
//      point that reaches a zero distance (the reference then passes over
//      that linestring, whose other segments may be unlisted) or none is
//      folded over every candidate.
// A group whose list overflows, or that meets a linestring outside the
// float32 frames, a non-finite point or an unusable grid, is left to the exact
// method's kernels, which spread it over several warps.  (Scanned by its own
// warp, 1081 points of sparse leaves x 3190 linestrings took 11.5 ms.)
__global__ void __launch_bounds__(kNearWarps * 32, 6)
  nearest_filtered_kernel(NearestArgs const a)
{
  __shared__ NearList s_list[kNearWarps];
  __shared__ uint16_t s_cand[kNearWarps][kNearCand][32];
  int const lane    = threadIdx.x & 31;
  NearList& L       = s_list[threadIdx.x >> 5];
  uint32_t const ng = *a.ngroups_p;
  bool const gok    = a.gf >= 1.17549435e-38f && a.gf < 1.0e30f;
  uint32_t nfb = 0, nscan = 0, nf64 = 0;
  float guess  = 0.0f;  // squared radius expected to hold the next group's list
  for (;;) {
    unsigned long long gg = 0;
    if (lane == 0) gg = atomicAdd(a.next_group, 1ull);
    uint64_t const gi = __shfl_sync(0xFFFFFFFFu, gg, 0);
    if (gi >= ng) break;
    uint32_t const k0   = a.group_start[gi];
    uint32_t const k1   = gi + 1 < ng ? a.group_start[gi + 1] : static_cast<uint32_t>(a.npairs);
    uint32_t const quad = a.pair_quad[k0];
    uint32_t const len  = a.qlen[quad];
    uint64_t const off  = a.qoff[quad];
    LeafFrame const lf  = a.frames[gi];
    bool listed         = !lf.nonfinite && gok;
    float mg            = 0.0f;
    float rad           = guess;  // squared radius of the list
    uint32_t n          = 0;
    if (listed) {
      n = list_segments(a, L, k0, k1, lf, rad, mg);
      if (n == kListOverflow && rad > 0.0f) {
        __syncwarp();
        rad = 0.0f;
        n   = list_segments(a, L, k0, k1, lf, rad, mg);
      }
      listed = n != kListOverflow && n != kListFrame;
      if (listed && n == 0) {
        // no segment within the radius: one from the chunks' vertices
        rad    = group_upper(a, k0, k1, lf);
        listed = rad < INFINITY;
        if (listed) {
          n      = list_segments(a, L, k0, k1, lf, rad, mg);
          listed = n != kListOverflow && n != kListFrame && n > 0;
        }
      }
    }
    if (listed) {
      float const dm  = 1.1920928955078125e-07f * mg;
      float const tol = 4.76837158203125e-07f * mg;
      float r2        = 0.0f;
      for (uint32_t c = lane; c < len; c += 32) {
        uint64_t const pos = off + c;
        if (pos >= a.npi) continue;
        float2 const uv = a.u[pos];
        float const U   = list_upper(L, n, uv.x, uv.y, dm, tol);
        r2              = fmaxf(r2, U);
        // kept for step 4 (the same lane reads it) where the distance will be
        *reinterpret_cast<float*>(a.od + pos) = U;
      }
      r2 = warp_max(r2);
      __syncwarp();  // every lane is done with the first list
      listed = r2 < INFINITY;
      if (listed) {
        float const need = r2 * 1.0000009536743164f;
        if (need > rad) {
          n      = list_segments(a, L, k0, k1, lf, need, mg);
          listed = n != kListOverflow && n != kListFrame && n > 0;
        }
        guess = fmaxf(0.7f * guess, 1.3f * need);
      }
    }
    if (!listed) {
      __syncwarp();
      if (lane == 0) {
        a.left[atomicAdd(a.nleft, 1u)] = static_cast<uint32_t>(gi);
        atomicAdd(a.nleft + 1, len);
      }
      ++nscan;
      continue;
    }
    float const dm  = 1.1920928955078125e-07f * mg;
    float const tol = 4.76837158203125e-07f * mg;
    uint16_t(&cand)[kNearCand][32] = s_cand[threadIdx.x >> 5];
    for (uint32_t c0 = 0; c0 < len; c0 += 32) {
      uint64_t const pos = off + c0 + static_cast<uint32_t>(lane);
      bool const act     = c0 + static_cast<uint32_t>(lane) < len && pos < a.npi;
      // this point's candidates: the listed segments whose estimate can
      // reach U, which starts at the bound of step 2 and shrinks on the way;
      // the first kNearCand of them are kept in list order
      float2 const uv = act ? a.u[pos] : make_float2(0.0f, 0.0f);
      float Uw        = 0.0f;
      uint32_t nc     = 0;
      if (act) {
        float U = *reinterpret_cast<float const*>(a.od + pos);
        Uw      = U * 1.0000000009313226f + 7.52316384526264e-37f;
        for (uint32_t t = 0; t < n; ++t) {
          float4 const e  = L.e[t];
          float4 const sb = make_float4(fminf(e.x, e.z), fminf(e.y, e.w), fmaxf(e.x, e.z),
                                        fmaxf(e.y, e.w));
          if (box_lb(uv.x, uv.y, sb, tol) > Uw) continue;
          float est, err;
          seg_estimate(uv.x, uv.y, e, dm, est, err);
          if (est - err > Uw) continue;
          U  = fminf(U, est + err);
          Uw = U * 1.0000000009313226f + 7.52316384526264e-37f;
          if (nc < kNearCand) cand[nc][lane] = static_cast<uint16_t>(t);
          ++nc;
        }
        if (nc > kNearCand) {
          // some may no longer reach the final bound: list them again
          nc = 0;
          for (uint32_t t = 0; t < n; ++t) {
            if (!seg_can_reach(L, t, uv.x, uv.y, dm, tol, Uw)) continue;
            if (nc < kNearCand) cand[nc][lane] = static_cast<uint16_t>(t);
            ++nc;
          }
        }
      }
      double px = 0.0, py = 0.0;
      if (act) a.src.load(pos, px, py);
      // The float64 distance of every candidate; per segment, since a
      // linestring's distance is the smallest of its segments' (square
      // roots are monotone) and the reference's winner is the smallest
      // non-zero (distance, id): the fold needs no order.  The lanes take
      // their r-th candidates together, so each float64 instruction serves
      // every lane that has one.  A segment at distance exactly 0 makes its
      // linestring's distance 0, which the reference passes over; such a
      // point is folded over every candidate instead.
      bool have = false, zero = false;
      uint32_t bid = 0;
      double bd    = 0.0;
      double bd2   = 0.0;  // smallest squared distance so far (its root is bd)
      auto fold_seg = [&](uint32_t t) {
        uint32_t const sg = L.seg[t];
        ++nf64;
        double const d2 =
          segment_dist2<double>(px, py, a.lx[sg], a.ly[sg], a.lx[sg + 1], a.ly[sg + 1]);
        if (!(d2 <= static_cast<double>(Uw))) return;
        if (d2 == 0.0) {
          zero = true;
          return;
        }
        // a squared distance more than 2^-48 above the smallest so far has a
        // larger (rounded) square root: it can neither win nor tie, so its
        // root is not needed
        if (have && d2 > bd2 * 1.0000000000000036) return;
        double const d     = sqrt(d2);
        uint32_t const lid = L.lid[t];
        if (!have || d < bd || (d == bd && lid < bid)) {
          bd  = d;
          bid = lid;
        }
        bd2  = have ? fmin(bd2, d2) : d2;
        have = true;
      };
      uint32_t const mine   = nc < kNearCand ? nc : kNearCand;
      uint32_t const rounds = __reduce_max_sync(0xFFFFFFFFu, mine);
      __syncwarp();  // every lane's candidates are stored
      for (uint32_t r = 0; r < rounds; ++r)
        if (r < mine && !zero) fold_seg(cand[r][lane]);
      if (nc > kNearCand && !zero) {
        // more candidates than kept: the rest in list order, this lane alone
        uint32_t seen = 0;
        for (uint32_t t = 0; t < n && !zero; ++t) {
          if (!seg_can_reach(L, t, uv.x, uv.y, dm, tol, Uw)) continue;
          if (seen++ < kNearCand) continue;
          fold_seg(t);
        }
      }
      __syncwarp();  // the candidate slots are reused by the next chunk
      fold_lanes(a, k0, k1, act && (!have || zero), px, py, have, bid, bd, nfb);
      if (act) {
        if (have) {
          a.opt[pos] = static_cast<uint32_t>(pos);
          a.ols[pos] = bid;
        }
        a.od[pos] = have ? bd : 0.0;
      }
    }
    __syncwarp();  // the next group rewrites this warp's list
  }
  if (a.stats) {
    for (int o = 16; o > 0; o >>= 1) {
      nfb += __shfl_xor_sync(0xFFFFFFFFu, nfb, o);
      nf64 += __shfl_xor_sync(0xFFFFFFFFu, nf64, o);
    }
    if (lane == 0 && nfb) atomicAdd(a.stats, static_cast<unsigned long long>(nfb));
    if (lane == 0 && nscan) atomicAdd(a.stats + 1, static_cast<unsigned long long>(nscan));
    if (lane == 0 && nf64) atomicAdd(a.stats + 3, static_cast<unsigned long long>(nf64));
  }
}

template <typename T>
void run(uint32_t const* pair_ls, uint32_t const* pair_quad, size_t npairs,
         cspt_quadtree const* tree, uint32_t const* point_indices, size_t npi, T const* x,
         T const* y, uint32_t const* lso, size_t nlso, T const* lx, T const* ly,
         cspt_method method, Allocator const& alloc, uint32_t* opt, uint32_t* ols, T* od,
         T const* ordered)
{
  cudaStream_t const s = alloc.stream();
  PointSource<T> const src{point_indices, x, y, ordered};
  init_rows_kernel<<<grid_for(npi, 256, sm_grid(16u)), 256, 0, s>>>(npi, opt, ols, od, sizeof(T));
  CSPT_CHECK_LAUNCH();
  // groups: runs of consecutive pairs with the same quadrant first-point offset
  uint32_t const* qoff = tree->offset;
  Buffer<uint32_t> gstart(alloc, npairs + 1);
  uint32_t* gs = gstart.data();
  scan_apply<uint32_t>(
    [pair_quad, qoff] __device__(size_t k) {
      return (k == 0 || qoff[pair_quad[k]] != qoff[pair_quad[k - 1]]) ? 1u : 0u;
    },
    [gs] __device__(size_t k, uint32_t e, uint32_t f) {
      if (f) gs[e] = static_cast<uint32_t>(k);
    },
    npairs, gs + npairs, alloc);
  size_t const nls = nlso > 0 ? nlso - 1 : 0;
  if constexpr (std::is_same<T, double>::value) {
    if (method == CSPT_METHOD_FILTERED) {
      // linestring index
      std::unique_ptr<KernelTimer> index_timer(new KernelTimer("nearest_index", s));
      Buffer<double4_16a> box(alloc, nls);
      Buffer<uint8_t> lexact(alloc, nls);
      Buffer<double> grid(alloc, 1);
      unsigned const lgrd = grid_for(nls * 32, 256, sm_grid(32u));
      ls_box_kernel<<<lgrd, 256, 0, s>>>(lso, nls, lx, ly, box.data(), lexact.data());
      CSPT_CHECK_LAUNCH();
      ls_grid_kernel<<<1, 1024, 0, s>>>(box.data(), nls, grid.data());
      CSPT_CHECK_LAUNCH();
      size_t const nv = nls ? read_back(lso + nls, s) : 0;
      Buffer<long long> aix(alloc, nls), aiy(alloc, nls);
      Buffer<float> maxoff(alloc, nls);
      size_t const slots = chunk_slots(nv, nls);
      size_t const sslots = super_slots(nv, nls);
      // (short of memory: without the exact kernels' boxes)
      size_t const bnls = alloc.frugal() ? 0 : nls, bslots = alloc.frugal() ? 0 : slots,
                   bnv  = alloc.frugal() ? 0 : nv;
      Buffer<float4> cbox(alloc, slots), seg32(alloc, nv), abs_ls(alloc, bnls),
        abs_chunk(alloc, bslots), sbox(alloc, sslots);
      Buffer<float2> vertex(alloc, bnv);
      Buffer<LsRec> lrec(alloc, nls);
      ls_fill_kernel<<<lgrd, 256, 0, s>>>(lso, nls, lx, ly, box.data(), grid.data(),
                                          lexact.data(), aix.data(), aiy.data(),
                                          maxoff.data(), cbox.data(), seg32.data(), lrec.data(),
                                          slots, abs_ls.data(), abs_chunk.data(), sslots, sbox.data(),
                                          static_cast<uint32_t>(bnv), vertex.data());
      CSPT_CHECK_LAUNCH();
      box.reset();
      double const g = read_back(grid.data(), s);
      index_timer.reset();
      // leaf frames of the groups
      Buffer<float2> u(alloc, npi);
      size_t const most = alloc.frugal() ? read_back(gs + npairs, s) : npairs;  // groups
      Buffer<LeafFrame> frames(alloc, most);
      std::unique_ptr<KernelTimer> frames_timer(new KernelTimer("leaf_frames", s));
      leaf_frame_kernel<<<grid_for(npairs * 32, 256, sm_grid(32u)), 256, 0, s>>>(
        gs, gs + npairs, pair_quad, tree->length, qoff, src, npi, grid.data(), u.data(),
        frames.data());
      CSPT_CHECK_LAUNCH();
      frames_timer.reset();
      LinestringIndexView liv{aix.data(),  aiy.data(),   maxoff.data(), cbox.data(),
                              sbox.data(), seg32.data(), lexact.data(), lrec.data()};
      LsBounds const bounds{abs_ls.data(), abs_chunk.data(), static_cast<uint32_t>(bslots),
                            vertex.data(), static_cast<uint32_t>(bnv)};
      // points folded whole, groups scanned, next group, float64 segment distances
      // (and the groups left and their points, as 32 bits)
      Buffer<unsigned long long> fb(alloc, 5);
      CSPT_CUDA_TRY(cudaMemsetAsync(fb.data(), 0, 5 * sizeof(unsigned long long), s));
      Buffer<uint32_t> left(alloc, most);
      uint32_t* const nleft = reinterpret_cast<uint32_t*>(fb.data() + 4);
      NearestArgs const na{gs,          gs + npairs,  npairs,     pair_ls,   pair_quad,
                           tree->length, qoff,        src,        npi,       lso,
                           nls,          lx,          ly,         u.data(),  frames.data(),
                           liv,          bounds,      static_cast<float>(g), opt, ols,    od,
                           fb.data(),    fb.data() + 2, left.data(), nleft};
      KernelTimer timer("nearest", s);
      int per_sm = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, nearest_filtered_kernel,
                                                        kNearWarps * 32, 0) != cudaSuccess ||
          per_sm < 1) {
        (void)cudaGetLastError();
        per_sm = 1;
      }
      nearest_filtered_kernel<<<grid_for(npairs * 32, kNearWarps * 32,
                                         sm_grid(static_cast<unsigned>(per_sm))),
                                kNearWarps * 32, 0, s>>>(na);
      CSPT_CHECK_LAUNCH();
      nearest_point_kernel<double><<<sm_grid(4u), 256, 0, s>>>(
        left.data(), nleft, gs, gs + npairs, npairs, kPointSplit, pair_quad, tree->length, qoff,
        src, npi, FoldArgs<double>{pair_ls, lso, nls, lx, ly, bounds}, opt, ols, od);
      CSPT_CHECK_LAUNCH();
      nearest_kernel<double><<<sm_grid(8u), 256, 0, s>>>(
        left.data(), nleft, gs, gs + npairs, npairs, kLaneSplit, pair_ls, pair_quad,
        tree->length, qoff, src, npi, lso, nls, lx, ly, bounds, opt, ols, od);
      CSPT_CHECK_LAUNCH();
      unsigned long long st[4];
      CSPT_CUDA_TRY(cudaMemcpyAsync(st, fb.data(), sizeof(st), cudaMemcpyDeviceToHost, s));
      CSPT_CUDA_TRY(cudaStreamSynchronize(s));
      last_fallbacks()     = st[0];
      last_group_scans()   = st[1];
      last_f64_segments()  = st[3];
      return;
    }
  }
  // the sizes of the launch and of the boxes, in one wait
  uint32_t h[2] = {0, 0};  // groups, vertices
  CSPT_CUDA_TRY(cudaMemcpyAsync(h, gs + npairs, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  if (nls)
    CSPT_CUDA_TRY(cudaMemcpyAsync(h + 1, lso + nls, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  CSPT_CUDA_TRY(cudaStreamSynchronize(s));
  bool const lean = alloc.frugal();  // without the boxes: every candidate is evaluated
  size_t const ng = h[0], slots = lean ? 0 : chunk_slots(h[1], nls);
  uint32_t const bnv = lean ? 0 : h[1];
  Buffer<float4> ls_box(alloc, lean ? 0 : nls), chunk_box(alloc, slots);
  Buffer<float2> vertex(alloc, bnv);
  LsBounds const bounds{ls_box.data(), chunk_box.data(), static_cast<uint32_t>(slots),
                        vertex.data(), bnv};
  if (!lean) {
    ls_bounds_kernel<T><<<grid_for(nls * 32, 256, sm_grid(32u)), 256, 0, s>>>(
      lso, nls, lx, ly, slots, ls_box.data(), chunk_box.data(), bnv, vertex.data());
    CSPT_CHECK_LAUNCH();
  }
  if (npi <= kWarpPoints) {
    KernelTimer timer("nearest", s);
    nearest_point_kernel<T><<<grid_for(npi * 32, 256, sm_grid(8u)), 256, 0, s>>>(
      nullptr, gs + npairs, gs, gs + npairs, npairs, kPointSplit, pair_quad, tree->length, qoff,
      src, npi,
      FoldArgs<T>{pair_ls, lso, nls, lx, ly, bounds}, opt, ols, od);
    CSPT_CHECK_LAUNCH();
  } else {
    KernelTimer timer("nearest", s);
    // warps per group: enough for 16 warps on every SM, at most kLaneSplit (a
    // leaf of 256 points has no more rounds of 32)
    size_t const fill    = static_cast<size_t>(num_sms()) * 16;
    uint32_t const split = static_cast<uint32_t>(
      ng == 0 ? 1 : std::min<size_t>(kLaneSplit, std::max<size_t>(1, fill / ng)));
    nearest_kernel<T><<<grid_for(ng * split * 32, 256, sm_grid(32u)), 256, 0, s>>>(
      nullptr, gs + npairs, gs, gs + npairs, npairs, split, pair_ls, pair_quad, tree->length, qoff,
      src, npi, lso, nls, lx, ly, bounds, opt, ols, od);
    CSPT_CHECK_LAUNCH();
  }
}

}  // namespace

void quadtree_point_to_nearest_linestring(uint32_t const* pair_ls, uint32_t const* pair_quad,
                                          size_t npairs, cspt_quadtree const* tree,
                                          uint32_t const* point_indices, size_t npi,
                                          void const* x, void const* y, uint32_t const* lso,
                                          size_t nlso, void const* lx, void const* ly,
                                          cspt_dtype dtype, cspt_method method,
                                          Allocator const& alloc, uint32_t* opt, uint32_t* ols,
                                          void* od, void const* ordered)
{
  if (dtype == CSPT_FLOAT64)
    run<double>(pair_ls, pair_quad, npairs, tree, point_indices, npi,
                static_cast<double const*>(x), static_cast<double const*>(y), lso, nlso,
                static_cast<double const*>(lx), static_cast<double const*>(ly), method, alloc,
                opt, ols, static_cast<double*>(od), static_cast<double const*>(ordered));
  else
    run<float>(pair_ls, pair_quad, npairs, tree, point_indices, npi, static_cast<float const*>(x),
               static_cast<float const*>(y), lso, nlso, static_cast<float const*>(lx),
               static_cast<float const*>(ly), method, alloc, opt, ols, static_cast<float*>(od),
               static_cast<float const*>(ordered));
}

}  // namespace cspt
