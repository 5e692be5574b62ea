// Unindexed point-in-polygon on sm_103a: every point against every polygon
// (at most 31, one result bit each), and the pairwise form (point i against
// polygon i).
//
// Reference: cpp/src/point_in_polygon/point_in_polygon.cu:36-150 (column API
// and validation), cpp/include/cuspatial/detail/point_in_polygon.cuh:41-140
// (pip_functor and the pairwise transform) and detail/algorithm/
// is_point_in_polygon.cuh:45-100 (the per-pair test).
//
// Bitmask form: the polygons go into the slab index (polygon_index.cuh), which
// limits each test to the edges of the point's slab; each lane holds one
// polygon's index fields in registers and the lanes of a warp cover
// (point, polygon) combinations.  With float64 input and the filtered method
// each point is placed once on the index's anchor grid (bit arithmetic, no
// float64 instruction) and the float32 filter decides each polygon, as in the
// quadtree join.
//
// Pairwise form: every polygon is used once, so no index is built; a warp
// walks the vertices of up to 32 consecutive polygons as one run, one vertex
// per lane, and combines the edge results per ring (on-edge OR, crossing
// parity XOR), which equals the reference's sequential walk wherever its
// skipped vertices are exact repeats (polygon_index.cuh, points 1 and 2);
// polygons where that can fail (non-finite or sub-2^-1019 coordinates) are
// walked sequentially by one lane.  With float64 input and the filtered
// method each vertex is moved into the point's frame in float32 on the
// integer and float32 pipes, and an edge takes the reference's float64
// expression only where the error bound below cannot decide it.
#include <algorithm>

#include "common.cuh"
#include "f32_split.cuh"
#include "pip_test.cuh"
#include "polygon_index.cuh"

namespace cspt {
namespace {

constexpr unsigned kPointsBlock = 256;

// Places v on the power-of-two grid 2^k, from its bit pattern: q = v / 2^k
// truncated toward zero, u = fl32(v - q 2^k).  False where the split is not
// representable (non-finite or subnormal v, |v - q 2^k| below 2^-120, q
// beyond 2^62); the caller then uses the exact test.
__device__ inline bool grid_split(double v, int k, long long& q, float& u)
{
  unsigned long long const b = static_cast<unsigned long long>(__double_as_longlong(v));
  int const e                = static_cast<int>((b >> 52) & 0x7FFull);
  unsigned long long m       = b & ((1ull << 52) - 1ull);
  bool const neg             = (b >> 63) != 0ull;
  if (e == 0x7FF) return false;
  if (e == 0) {
    q = 0;
    u = 0.0f;
    return m == 0ull;  // +-0 only
  }
  m |= 1ull << 52;
  int const e2 = e - 1075;  // v = +-m 2^e2
  if (e2 < -120) return false;
  unsigned long long qq = 0, low = 0;
  if (e2 >= k) {
    if (e2 - k > 9) return false;
    qq = m << (e2 - k);
  } else {
    int const sh = k - e2;
    if (sh >= 64) {
      low = m;
    } else {
      qq  = m >> sh;
      low = m & ((1ull << sh) - 1ull);
    }
  }
  // low < 2^(k - e2): |u| < 2^k, and scaling by 2^e2 (>= 2^-120) is exact
  float const f = low ? __ull2float_rn(low) * __int_as_float((e2 + 127) << 23) : 0.0f;
  q             = neg ? -static_cast<long long>(qq) : static_cast<long long>(qq);
  u             = neg ? -f : f;
  return true;
}

// Bitmask form (pip_functor, detail/point_in_polygon.cuh:41-66): bit p of
// out[i] = point i inside polygon p.  With at most 31 polygons every lane
// keeps one polygon's index fields in registers for the whole kernel: with
// P = 2^lp >= the polygon count, lane = (slot s, polygon p) with
// p = lane % P and s = lane / P, so a warp tests 32 / P points at a time
// against all polygons; a ballot then holds each point's mask in P bits.
// Points are read (and masks written) 32 at a time, one per lane, and passed
// to the testing lanes by shuffles.
template <typename T, bool Filtered>
__global__ void __launch_bounds__(kPointsBlock)
  points_pip_kernel(T const* __restrict__ x, T const* __restrict__ y, size_t n,
                    PolygonIndexView<T> ix, T bounds_share, uint32_t lp,
                    int32_t* __restrict__ out, unsigned long long* __restrict__ refined)
{
  // (bounds_share > 0: the index may carry bounds instead, for the grid of cells)
  if (bounds_share > T{0} && has_bounds(ix.origin, bounds_share)) return;
  int const lane       = threadIdx.x & 31;
  uint32_t const P     = 1u << lp;
  uint32_t const S     = 32u >> lp;
  uint32_t const p     = static_cast<uint32_t>(lane) & (P - 1u);
  uint32_t const slot  = static_cast<uint32_t>(lane) >> lp;
  unsigned const pbits = P == 32u ? 0xFFFFFFFFu : ((1u << P) - 1u);
  bool const has_poly  = p < ix.num_polygons;
  uint32_t nref        = 0;
  // the lane's polygon
  float4 box    = make_float4(0.f, 0.f, 0.f, 0.f);
  float mp = 0.0f, invh = 0.0f, gf = 0.0f;
  uint32_t ns = 1, slab0 = 0, vb = 0, ve = 0;
  long long aix = 0, aiy = 0;
  bool exact_poly = true, gok = false;
  int gk          = 0;
  if constexpr (Filtered) {
    double const g = *ix.grid;
    gf             = static_cast<float>(g);
    gok            = gf >= 1.17549435e-38f && gf < 1.0e30f;  // normal float grid step
    gk = static_cast<int>((static_cast<unsigned long long>(__double_as_longlong(g)) >> 52) &
                          0x7FFull) -
         1023;
    if (has_poly) {
      box        = ix.box32[p];
      mp         = ix.max_offset[p];
      invh       = ix.inv_slab_h32[p];
      ns         = ix.num_slabs[p];
      slab0      = ix.slab_base[p];
      vb         = ix.vert_begin[p];
      ve         = ix.vert_end[p];
      aix        = ix.anchor_ix[p];
      aiy        = ix.anchor_iy[p];
      exact_poly = ix.exact_only[p] != 0;
    }
  }
  size_t const warp   = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5;
  size_t const nwarps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  for (size_t base = warp * 32; base < n; base += nwarps * 32) {
    size_t const i = base + static_cast<size_t>(lane);
    T px = T{0}, py = T{0};
    if (i < n) {
      px = x[i];
      py = y[i];
    }
    long long qx = 0, qy = 0;
    float ux = 0.0f, uy = 0.0f;
    bool framed = false;
    if constexpr (Filtered)
      framed = gok && grid_split(px, gk, qx, ux) && grid_split(py, gk, qy, uy);
    int32_t mine = 0;
    for (uint32_t b = 0; b < P; ++b) {
      int const src  = static_cast<int>(b * S + slot);  // lane holding the tested point
      T const tx     = __shfl_sync(0xFFFFFFFFu, px, src);
      T const ty     = __shfl_sync(0xFFFFFFFFu, py, src);
      bool const live = has_poly && base + static_cast<size_t>(src) < n;
      bool hit        = false;
      if constexpr (Filtered) {
        long long const tqx = __shfl_sync(0xFFFFFFFFu, qx, src);
        long long const tqy = __shfl_sync(0xFFFFFFFFu, qy, src);
        float const tux     = __shfl_sync(0xFFFFFFFFu, ux, src);
        float const tuy     = __shfl_sync(0xFFFFFFFFu, uy, src);
        bool const tfr      = __shfl_sync(0xFFFFFFFFu, static_cast<int>(framed), src) != 0;
        if (live) {
          long long const dix = aix - tqx;
          long long const diy = aiy - tqy;
          bool const exact    = !tfr || exact_poly || dix <= -16777216LL || dix >= 16777216LL ||
                             diy <= -16777216LL || diy >= 16777216LL;
          if (exact) {
            ++nref;
            hit = pip_exact<double>(tx, ty, ix, p);
          } else {
            // anchor offset in grid steps: exact in float32 below 2^24 steps
            float const dx = static_cast<float>(static_cast<int>(dix)) * gf;
            float const dy = static_cast<float>(static_cast<int>(diy)) * gf;
            hit            = filtered_test<false>(
              ix, p, tux - dx, tuy - dy, mp, fmaxf(fabsf(tux), fabsf(tuy)), box, invh, 0.0f, ns,
              slab0, vb, ve,
              [&](double& ox, double& oy) {
                ox = tx;
                oy = ty;
              },
              nref);
          }
        }
      } else {
        if (live) hit = pip_exact<T>(tx, ty, ix, p);
      }
      unsigned const bal = __ballot_sync(0xFFFFFFFFu, hit);
      uint32_t const own = static_cast<uint32_t>(lane) - b * S;  // this lane's point slot
      if (own < S) mine = static_cast<int32_t>((bal >> (own * P)) & pbits);
    }
    if (i < n) out[i] = mine;
  }
  if (Filtered && refined) {
    for (int o = 16; o > 0; o >>= 1) nref += __shfl_xor_sync(0xFFFFFFFFu, nref, o);
    if (lane == 0 && nref) atomicAdd(refined, static_cast<unsigned long long>(nref));
  }
}

// ---------------------------------------------------------------------------
// Bitmask form on many float64 points (either method): a grid of cells over the
// polygons' boxes, each cell holding for every polygon whether its points are
// inside, outside, or have to be tested (two bit words), so that a point costs
// one 8-byte lookup for all polygons.
//
// A cell decides a polygon when no edge meets the cell and no exactly vertical
// edge has its x in the cell's x-range.  An edge's box (outward_box) beyond the
// cell, or its line further from the cell's centre than the cell reaches, by
// margins above the float32 roundings here and the float64 ones of the
// reference, means that the reference decides the edge correctly for every point
// of the cell; and a region that no edge of the closed rings enters lies on one
// side of them, so all its points have the centre's result.  A cell's rectangle
// is widened to hold every point that the float32 lookup sends there, with the
// points' own bounds.  Points beyond the polygons' common box are outside all of
// them.  Polygons that are walked with the reference loop, and points beyond
// float32, are tested.
//
// The cells cost one classification per polygon for every kPointsPerCell
// points; the points read 16 and write 4 bytes, and the tests that remain are
// queued per warp so that they run with full warps.
// 10M points x 31 polygons of 100 sides: 1612 us testing every polygon whose box
// holds the point (bound by the L1 wavefronts of the slab reads; a warp queue
// for full warps alone gave 1620 to 1800 us); 102 us for the cells and 129 for
// the points with the grid, the call 1757 -> 328 us (exact 12.2 ms -> 318 us).
// With edges told apart by their boxes alone the points took 367 us.
// ---------------------------------------------------------------------------
constexpr int kPointSets        = 4;   // rounds of 32 points a warp takes together
// (8 / 16 / 32 points a cell, 31 polygons: 10M points 590 / 336 / 340 us a call,
// 300k points of 1000 sides - / 181 / 195)
constexpr size_t kPointsPerCell = 16;
constexpr uint32_t kGridMin = 32, kGridMax = 1024;  // cells along an axis
constexpr uint32_t kRowEntries = 512;  // entries of a polygon that any row streams

struct CellPoly {
  float4 box;  // outward
  float my, y0, invh, inner;
  uint32_t ns, slab0, vb, ve;
};
struct CellGrid {
  float x0, y0, x1, y1;  // common box (outward)
  float iw, ih;          // cells per unit
  uint32_t walked;       // polygons tested for every point
};

// Loads the polygons' fields and the grid's geometry into shared memory.
__device__ inline void load_cells(PolygonIndexView<double> const& ix, uint32_t g,
                                  CellPoly (&s_poly)[32], CellGrid& s_grid)
{
  if (threadIdx.x < 32) {
    uint32_t const p = threadIdx.x;
    bool const have  = p < ix.num_polygons;
    float4 b = make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY);
    bool walk = false;
    if (have) {
      // (a polygon without vertices keeps the empty box; one beyond float32 is
      // tested for every point, so that the others keep a finite grid)
      bool const empty = ix.pminx[p] > ix.pmaxx[p];
      float4 const v   = ix.box32[p];
      walk = ix.exact_only[p] != 0 || (!empty && !(v.z - v.x < INFINITY && v.w - v.y < INFINITY));
      CellPoly f{};
      f.box   = walk || empty ? b : v;
      f.my    = fmaxf(fabsf(f.box.y), fabsf(f.box.w));
      f.inner = __fmaf_ru(f.my, 9.5367431640625e-07f, 1.0e-36f);  // 2^-20
      f.y0    = truncated_f32(ix.pminy[p] - ix.origin[1]);
      f.invh  = ix.inv_slab_h32[p];
      f.ns    = ix.num_slabs[p];
      f.slab0 = ix.slab_base[p];
      f.vb    = ix.vert_begin[p];
      f.ve    = ix.vert_end[p];
      s_poly[p] = f;
      b         = f.box;
    }
    for (int o = 16; o > 0; o >>= 1) {
      b.x = fminf(b.x, __shfl_xor_sync(0xFFFFFFFFu, b.x, o));
      b.y = fminf(b.y, __shfl_xor_sync(0xFFFFFFFFu, b.y, o));
      b.z = fmaxf(b.z, __shfl_xor_sync(0xFFFFFFFFu, b.z, o));
      b.w = fmaxf(b.w, __shfl_xor_sync(0xFFFFFFFFu, b.w, o));
    }
    unsigned const walked = __ballot_sync(0xFFFFFFFFu, walk);
    if (threadIdx.x == 0)
      s_grid = CellGrid{b.x, b.y, b.z, b.w, static_cast<float>(g) / (b.z - b.x),
                        static_cast<float>(g) / (b.w - b.y), walked};
  }
  __syncthreads();
}

// The cell of coordinate t along an axis (monotone in t).
__device__ inline uint32_t cell_along(float t, float origin, float per_unit, uint32_t g)
{
  float const f = (t - origin) * per_unit;
  if (!(f > 0.0f)) return 0u;
  return f >= static_cast<float>(g) ? g - 1u : min(static_cast<uint32_t>(f), g - 1u);
}
// Bounds of the points of cell c along an axis, ends included: the lookup is
// off by less than g 2^-22 cells, and a point lies within outward_width of
// its float32 value.
__device__ inline void cell_range(uint32_t c, float origin, float end, float per_unit, float& lo,
                                  float& hi)
{
  float const w     = 1.0f / per_unit;
  float const slack = 3.0f * outward_width(fmaxf(fabsf(origin), fabsf(end))) + 0.0009765625f * w;
  lo = origin + static_cast<float>(c) * w - slack;
  hi = origin + static_cast<float>(c + 1u) * w + slack;
}

// An edge whose box meets the cell: 2 when the edge may meet the cell or the
// centre's result is not certain, 1 when the centre sees it as a toggle, else 0.
// (cx, cy) the centre, (hw, hh) half the cell, m the largest coordinate.
// Truncated coordinates (relative to the index's origin, as all here) are off by
// 2^-23 m, their differences by less than 2^-21 m, the cross product by less than 2^-20 m times the differences' sum.
__device__ inline int edge_by_line(PolygonIndexView<double> const& ix, uint32_t k, float4 const& e,
                                   float cx, float cy, float hw, float hh, float m, float inner)
{
  float4 const t = ix.edge32[ix.slab_edges[k] & kEntryVertex];
  float const ex = t.z - t.x, ey = t.w - t.y;
  float const dx = cx - t.x, dy = cy - t.y;
  float const cr    = __fmaf_rn(dx, ey, -(dy * ex));
  float const reach = __fmaf_rn(hw, fabsf(ey), hh * fabsf(ex));
  float const err   = 3.814697265625e-06f * m * (fabsf(ex) + fabsf(ey) + fabsf(dx) + fabsf(dy));
  // (an infinite cross product tells nothing, as in edge_by_side)
  if (!(fabsf(cr) > 1.001f * reach + err + 1.0e-36f && fabsf(cr) < INFINITY)) return 2;
  if (cy > e.w || cy < e.y) return 0;
  if (!(cy > e.y + inner && cy < e.w - inner)) return 2;
  return (cr < 0.0f) == (ey > 0.0f) ? 1 : 0;
}

// A lane per cell of a row, 32 cells a warp: the entries of the row's slabs are
// the same for all lanes.  `share` warps split the cells' polygons, as many as
// fill the GPU (a warp's chain of polygons, each a few dependent loads, bounds
// the kernel).  cells[row g + column] |= (inside, test), zero before.
__global__ void __launch_bounds__(kPointsBlock)
  points_cells_kernel(PolygonIndexView<double> ix, double bounds_share, uint32_t g,
                      uint32_t share, uint2* __restrict__ cells)
{
  if (bounds_share > 0.0 && !has_bounds(ix.origin, bounds_share)) return;
  constexpr unsigned kAll = 0xFFFFFFFFu;
  __shared__ CellPoly s_poly[32];
  __shared__ CellGrid grid;
  load_cells(ix, g, s_poly, grid);
  double const ox       = ix.origin[0];
  uint32_t const npoly  = static_cast<uint32_t>(ix.num_polygons);
  uint32_t const lane   = threadIdx.x & 31u;
  uint32_t const warps  = gridDim.x * (kPointsBlock / 32);
  uint32_t const perrow = g / 32u;
  for (uint32_t w = (blockIdx.x * kPointsBlock + threadIdx.x) >> 5; w < g * perrow * share;
       w += warps) {
    uint32_t const seg = w / share;
    uint32_t const row = seg / perrow, col = (seg - row * perrow) * 32u + lane;
    float xl, xu, yl, yu;
    cell_range(col, grid.x0, grid.x1, grid.iw, xl, xu);
    cell_range(row, grid.y0, grid.y1, grid.ih, yl, yu);
    float const cx = 0.5f * (xl + xu), cy = 0.5f * (yl + yu);
    float const hw = 0.5f * (xu - xl), hh = 0.5f * (yu - yl);
    float const mc = fmaxf(fmaxf(fabsf(xl), fabsf(xu)), fmaxf(fabsf(yl), fabsf(yu)));
    uint32_t inside = 0, test = 0;
    for (uint32_t p = w - seg * share; p < npoly; p += share) {
      CellPoly const& f = s_poly[p];
      if ((grid.walked >> p) & 1u) continue;
      if (yl > f.box.w || yu < f.box.y) continue;  // the row lies beyond the polygon
      bool const open = !(xl > f.box.z || xu < f.box.x);  // still to be decided
      if (!__any_sync(kAll, open)) continue;
      // (a row that holds the polygon's whole height decides nothing)
      bool meets = !((f.my + fmaxf(fabsf(yl), fabsf(yu))) * f.invh <= 16384.0f) ||
                   (yl <= f.box.y && yu >= f.box.w);
      if (f.vb < f.ve && !meets) {
        uint32_t lo = f.vb, hi = f.ve;
        while (lo < hi) {
          uint32_t const mid = (lo + hi) >> 1;
          if (ix.vert_x[mid] - ox < static_cast<double>(xl))
            lo = mid + 1;
          else
            hi = mid;
        }
        meets = lo < f.ve && ix.vert_x[lo] - ox <= static_cast<double>(xu);
      }
      bool in = false;
      if (__any_sync(kAll, open && !meets)) {
        float const m = fmaxf(mc, fmaxf(f.my, fmaxf(fabsf(f.box.x), fabsf(f.box.z))));
        uint32_t const j0 = slab_lookup(yl, f.y0, f.invh, f.ns),
                       j1 = slab_lookup(yu, f.y0, f.invh, f.ns),
                       jc = slab_lookup(cy, f.y0, f.invh, f.ns);
        uint32_t const E0 = ix.slab_start[f.slab0 + j0], E1 = ix.slab_start[f.slab0 + j1 + 1];
        uint32_t const C0 = ix.slab_start[f.slab0 + jc], C1 = ix.slab_start[f.slab0 + jc + 1];
        uint32_t const all = ix.slab_start[f.slab0 + f.ns] - ix.slab_start[f.slab0];
        // (a row that holds much of a large polygon decides little: 31 polygons of 1000
        // sides one cell wide, 200k points, exact: 948 us with its entries streamed, 313
        // without, 663 without the grid)
        bool const many = E1 - E0 > kRowEntries && E1 - E0 > all / 8u;
        if (many) meets = true;
#pragma unroll 4
        for (uint32_t k = many ? E1 : E0; k < E1; ++k) {
          float4 const e = ix.slab_e32[k];
          bool const near = !(xl > e.z || xu < e.x || yl > e.w || yu < e.y);
          // (beyond the cell's box the centre sees it left, right, above or below)
          int const d = near ? edge_by_line(ix, k, e, cx, cy, hw, hh, m, f.inner)
                             : edge_by_bounds(e, cx, cy, cx, cy, f.inner);
          bool const centre = k >= C0 && k < C1;
          meets |= d == 2 && (near || centre);
          in ^= d == 1 && centre;
        }
      }
      if (open) {
        if (meets)
          test |= 1u << p;
        else if (in)
          inside |= 1u << p;
      }
    }
    uint2* const cell = cells + static_cast<size_t>(row) * g + col;
    if (inside) atomicOr(&cell->x, inside);
    if (test) atomicOr(&cell->y, test);
  }
}

__global__ void __launch_bounds__(kPointsBlock)
  points_grid_kernel(double const* __restrict__ x, double const* __restrict__ y, size_t n,
                     PolygonIndexView<double> ix, double bounds_share, uint32_t g,
                     uint2 const* __restrict__ cells, uint32_t sets, int32_t* __restrict__ out,
                     unsigned long long* __restrict__ refined)
{
  if (bounds_share > 0.0 && !has_bounds(ix.origin, bounds_share)) return;
  constexpr unsigned kAll = 0xFFFFFFFFu;
  constexpr int kWarps = kPointsBlock / 32, kPts = 32 * kPointSets;
  __shared__ CellPoly s_poly[32];
  __shared__ CellGrid grid;
  __shared__ uint32_t s_mask[kWarps][kPts];
  __shared__ uint16_t s_queue[kWarps][64];  // point of the warp | polygon << 7
  static_assert(kPts == 128, "queue entries hold 7 bits of point");
  load_cells(ix, g, s_poly, grid);
  double const ox = ix.origin[0], oy = ix.origin[1];
  int const lane       = threadIdx.x & 31;
  int const warp       = threadIdx.x >> 5;
  unsigned const lt    = (1u << lane) - 1u;
  uint32_t const all   = static_cast<uint32_t>((1ull << ix.num_polygons) - 1ull);
  uint32_t nref        = 0;
  size_t const w0      = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5;
  size_t const nwarps  = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  size_t const per     = static_cast<size_t>(sets) * 32;
  for (size_t base = w0 * per; base < n; base += nwarps * per) {
    // tests queue entries [at, at + m), one per lane
    auto test = [&](uint32_t at, uint32_t m) {
      __syncwarp();
      if (static_cast<uint32_t>(lane) < m) {
        uint32_t const q    = s_queue[warp][at + lane];
        uint32_t const slot = q & (kPts - 1), p = q >> 7;
        CellPoly const& f   = s_poly[p];
        double const px = x[base + slot], py = y[base + slot];
        float const tx = truncated_f32(px - ox), ty = truncated_f32(py - oy);
        float const wx = outward_width(tx), wy = outward_width(ty);
        bool hit;
        if (((grid.walked >> p) & 1u) || !(f.my < INFINITY)) {  // (or without vertices)
          ++nref;
          hit = pip_exact<double>(px, py, ix, p);
        } else {
          auto const load = [&](double& a, double& b) {
            a = px;
            b = py;
          };
          bool const lookup = (f.my + fabsf(ty)) * f.invh <= 16384.0f;
          hit = bounds_test(ix, tx, ty, __fsub_rd(tx, wx), __fsub_rd(ty, wy), __fadd_ru(tx, wx),
                            __fadd_ru(ty, wy), f.inner,
                            1.001f * fmaxf(f.my, fmaxf(fabsf(f.box.x), fabsf(f.box.z))),
                            f.slab0 + bounds_slab(ix, p, lookup, ty, f.y0, f.invh, f.ns, load),
                            f.vb, f.ve, load, nref);
        }
        if (hit) atomicOr(&s_mask[warp][slot], 1u << p);
      }
      __syncwarp();
    };
    uint32_t queued = 0;
    // every round's points are loaded first, then their cells
    float2 t[kPointSets];
    uint2 cell[kPointSets];
#pragma unroll
    for (int r = 0; r < kPointSets; ++r) {
      size_t const i = base + r * 32 + lane;
      bool const have = static_cast<uint32_t>(r) < sets && i < n;
      t[r] = have ? make_float2(truncated_f32(x[i] - ox), truncated_f32(y[i] - oy))
                  : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < kPointSets; ++r) {
      size_t const i = base + r * 32 + lane;
      cell[r]        = make_uint2(0u, 0u);
      if (static_cast<uint32_t>(r) < sets && i < n) {
        float const wx = outward_width(t[r].x), wy = outward_width(t[r].y);
        if (!(wx < INFINITY && wy < INFINITY))
          cell[r].y = all;  // beyond float32 or not finite
        else if (__fsub_rd(t[r].x, wx) > grid.x1 || __fadd_ru(t[r].x, wx) < grid.x0 ||
                 __fsub_rd(t[r].y, wy) > grid.y1 || __fadd_ru(t[r].y, wy) < grid.y0)
          cell[r].y = grid.walked;
        else {
          cell[r] = cells[static_cast<size_t>(cell_along(t[r].y, grid.y0, grid.ih, g)) * g +
                          cell_along(t[r].x, grid.x0, grid.iw, g)];
          cell[r].y |= grid.walked;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kPointSets; ++r) {
      uint32_t const slot = r * 32 + lane;
      s_mask[warp][slot]  = cell[r].x;
      uint32_t left       = cell[r].y;
      for (;;) {
        unsigned const m = __ballot_sync(kAll, left != 0u);
        if (m == 0u) break;
        if (__popc(m) < 8) {
          // few points left: all polygons of one, a lane per polygon
          int const src       = __ffs(m) - 1;
          uint32_t const bits = __shfl_sync(kAll, left, src);
          if (lane == src) left = 0u;
          if ((bits >> lane) & 1u)
            s_queue[warp][queued + __popc(bits & lt)] =
              static_cast<uint16_t>((r * 32 + src) | (lane << 7));
          queued += __popc(bits);
          if (queued >= 32u) {
            queued -= 32u;
            test(queued, 32u);
          }
          continue;
        }
        if (left) {
          uint32_t const p = __ffs(left) - 1;
          left &= left - 1u;
          s_queue[warp][queued + __popc(m & lt)] = static_cast<uint16_t>(slot | (p << 7));
        }
        queued += __popc(m);
        if (queued >= 32u) {
          queued -= 32u;
          test(queued, 32u);
        }
      }
    }
    if (queued) test(0u, queued);
    __syncwarp();
    for (uint32_t r = 0; r < sets; ++r) {
      size_t const i = base + r * 32 + lane;
      if (i < n) out[i] = static_cast<int32_t>(s_mask[warp][r * 32 + lane]);
    }
    __syncwarp();
  }
  if (refined) {
    for (int o = 16; o > 0; o >>= 1) nref += __shfl_xor_sync(kAll, nref, o);
    if (lane == 0 && nref) atomicAdd(refined, static_cast<unsigned long long>(nref));
  }
}

__device__ inline bool same_bits(double a, double b)
{
  unsigned long long const u = __double_as_longlong(a), v = __double_as_longlong(b);
  return u == v || ((u | v) << 1) == 0ull;  // equal bits, or +0 and -0
}
__device__ inline bool same_bits(float a, float b) { return a == b; }
// exponent field <= 3: |a| < 2^-1019 (double), 2^-123 (float)
__device__ inline bool tiny_bits(double a)
{
  return ((static_cast<unsigned long long>(__double_as_longlong(a)) >> 52) & 0x7FFull) <= 3ull;
}
__device__ inline bool tiny_bits(float a) { return ((__float_as_uint(a) >> 23) & 0xFFu) <= 3u; }

// Pairwise form: a warp takes `per_warp` consecutive (point, polygon) pairs.
// Their polygons' vertices are one contiguous run, which the warp walks 32
// vertices at a time, one per lane, whatever the sizes of the rings in it: no
// lane waits for a larger polygon, and every load is coalesced.  The rings
// come 32 at a time, one per lane (vertex range, its point's offset parts,
// its closing vertex); a vertex finds its ring by counting ring starts, and
// the chunk's toggles and on-edge hits go back to the rings as ballots.
//
// Filtered (float64 input): a vertex coordinate minus the point's is taken
// from the float32 parts of both (f32_split.cuh):
//   f = (hi_v - hi_p) + (lo_v - lo_p),  |f - (v - p)| <= 2^-23 |f| + 2^-44 (|v| + |p|)
// (three float32 roundings and the parts left out).  Per edge, with
// m = max |f| of its two ends on an axis and p's coordinate there,
//   t = 2^-20 m + 2^-41 |p| + 2^-60
// is more than 4 times that error (|v| <= |p| + 1.01 m).
//   * Both y offsets beyond t_y: the y-flags (ay > py) are their signs.
//   * Same flags: the edge cannot toggle, and can be on the point only if it
//     is within 2^-48 |rise| of py (it is not: t_y >= 2^-21 |rise|) or exactly
//     vertical at px; with one x offset beyond t_x it is not vertical there.
//   * Flags differ and both x offsets beyond t_x on one side: px is outside
//     the edge's x-range, so it is not on the edge, and the reference's
//     comparison of lhs = (px - ax)(by - ay) with rhs = (bx - ax)(py - ay) has
//     |px - ax| >= |bx - ax| + t_x on the right of both (or a sign that
//     decides) and |by - ay| >= |py - ay| + t_y, far beyond its roundings:
//     toggles exactly when px is left of the edge.
//   * Flags differ otherwise: cr = a_y b_x - a_x b_y in float32 against
//     eb = 2 (t_x (|a_y| + |b_y|) + t_y (|a_x| + |b_x|)), above the offsets'
//     errors, float32's roundings (2^-23 of each product) and float64's.  Offsets
//     from about 2^64 on have products beyond float32: an infinite cr decides
//     nothing (eb, 2^-20 of them, may still be finite).
// Anything else, and any vertex with a coordinate that does not split (zero,
// below 2^-100, 2^100 and above, non-finite), takes the reference's float64
// edge test, which also finds the polygons that need the sequential walk
// (non-finite or sub-2^-1019 coordinates): its skip rule can differ only
// where a coordinate is below 2^-1019.
//
// 1M pairs of 4..400 vertices (9.4e7 vertices, 1.56 GB): 3.37 ms with a
// float64 subtraction and conversion per coordinate (float64 pipe 83% busy)
// and 8 lanes per polygon, 0.61 ms this way (2.5 TB/s; bound by instruction
// issue and the vertex loads: without the next chunk's loads in flight 1.18).
// Five resident blocks of 256 measured fastest: 0.99 / 0.71 / 0.64 / 0.61 ms
// with 2 / 3 / 4 / 5.  Exact float64: 7.8 -> 2.9 ms, float32 1.36 -> 0.50.
template <typename T, bool Filtered>
__global__ void __launch_bounds__(kPointsBlock, 5)
  pairwise_pip_kernel(T const* __restrict__ x, T const* __restrict__ y, size_t n,
                      uint32_t const* __restrict__ po, uint32_t const* __restrict__ ro,
                      T const* __restrict__ vx, T const* __restrict__ vy, uint32_t per_warp,
                      uint8_t* __restrict__ out, unsigned long long* __restrict__ refined)
{
  constexpr unsigned kAll = 0xFFFFFFFFu;
  // what a lane keeps of a vertex: its float32 offset, or the vertex itself
  using V                 = typename std::conditional<Filtered, float, T>::type;
  unsigned const lane     = threadIdx.x & 31;
  unsigned const le       = kAll >> (31u - lane);  // this lane and those below
  size_t const warp       = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5;
  size_t const nwarps     = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  uint32_t nref           = 0;
  for (size_t base = warp * per_warp; base < n; base += nwarps * per_warp) {
    uint32_t const np = n - base < per_warp ? static_cast<uint32_t>(n - base) : per_warp;
    // lane p: pair base + p
    bool const have_p = lane < np;
    size_t const i    = base + (have_p ? lane : np - 1);
    T const px = x[i], py = y[i];
    uint32_t const r0 = po[i], r1 = po[i + 1];
    bool literal = !(isfinite(px) && isfinite(py));
    bool on = false, within = false;
    F32Pair fx{0.0f, 0.0f}, fy{0.0f, 0.0f};
    if constexpr (Filtered) {
      // a point coordinate of 0 is its own parts; others that do not split
      // make every edge undecided
      float const nan = __int_as_float(0x7FC00000);
      if (px != T{0}) fx = splits_f32(px) ? split_f32(px) : F32Pair{nan, nan};
      if (py != T{0}) fy = splits_f32(py) ? split_f32(py) : F32Pair{nan, nan};
    }
    uint32_t const rb = __shfl_sync(kAll, r0, 0);
    uint32_t const re = __shfl_sync(kAll, r1, static_cast<int>(np - 1));
    for (uint32_t rr = rb; rr < re; rr += 32) {
      // lane j: ring rr + j, vertices [s, e)
      uint32_t const nr = re - rr < 32u ? re - rr : 32u;
      uint32_t const r  = rr + (lane < nr ? lane : nr - 1u);
      uint32_t const e  = ro[r + 1];
      uint32_t const s  = lane < nr ? ro[r] : e;
      // the pair holding the ring: the first whose rings end beyond it
      uint32_t pl = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        uint32_t const v = __shfl_sync(kAll, r1, static_cast<int>(pl) + step - 1);
        if (v <= r && pl + step < np) pl += step;
      }
      F32Pair qx{}, qy{};
      T rpx{}, rpy{};
      if constexpr (Filtered) {
        qx = F32Pair{__shfl_sync(kAll, fx.hi, pl), __shfl_sync(kAll, fx.lo, pl)};
        qy = F32Pair{__shfl_sync(kAll, fy.hi, pl), __shfl_sync(kAll, fy.lo, pl)};
      } else {
        rpx = __shfl_sync(kAll, px, pl);
        rpy = __shfl_sync(kAll, py, pl);
      }
      // the vertex, or its offset from the point with parts (ox, oy): NaN
      // where the vertex does not split
      auto keep = [](T ax, T ay, F32Pair const& ox, F32Pair const& oy, V& fa, V& fb) {
        if constexpr (Filtered) {
          F32Pair const a = split_f32(ax), b = split_f32(ay);
          bool const ok   = splits_f32(ax) && splits_f32(ay);
          float const nan = __int_as_float(0x7FC00000);
          fa              = ok ? (a.hi - ox.hi) + (a.lo - ox.lo) : nan;
          fb              = ok ? (b.hi - oy.hi) + (b.lo - oy.lo) : nan;
        } else {
          fa = ax;
          fb = ay;
        }
      };
      // the edge into a ring's first vertex starts at its last
      V zx{}, zy{};
      if (e > s) keep(vx[e - 1], vy[e - 1], qx, qy, zx, zy);
      bool rpar = false, ron = false, rlit = false;
      uint32_t const vb   = __shfl_sync(kAll, s, 0);
      uint32_t const ve   = __shfl_sync(kAll, e, static_cast<int>(nr - 1));
      bool const empties  = __any_sync(kAll, lane < nr && e <= s);
      uint32_t before     = 0;  // rings that start before the chunk
      V cx{}, cy{};                // the vertex before the chunk
      // the next chunk's vertices are loaded while this one's are tested
      T nx = vb + lane < ve ? vx[vb + lane] : T{1};
      T ny = vb + lane < ve ? vy[vb + lane] : T{1};
      for (uint32_t c = vb; c < ve; c += 32) {
        uint32_t const v = c + lane;
        bool const own   = v < ve;
        T const ax = nx, ay = ny;
        bool const more = ve - c > 32u && v + 32u < ve;
        nx              = more ? vx[v + 32u] : T{1};
        ny              = more ? vy[v + 32u] : T{1};
        // the vertex's ring
        uint32_t const d   = s - c;
        unsigned const beg = __reduce_or_sync(kAll, (d < 32u && e > s) ? 1u << d : 0u);
        int k              = static_cast<int>(before + __popc(beg & le)) - 1;
        if (empties) {
          k = 0;
#pragma unroll
          for (int step = 16; step > 0; step >>= 1) {
            uint32_t const q = __shfl_sync(kAll, e, k + step - 1);
            if (q <= v && k + step < 32) k += step;
          }
        }
        before += __popc(beg);
        bool und = own, tog = false, hit = false, lit = false;
        F32Pair ox{}, oy{};
        if constexpr (Filtered) {
          ox = F32Pair{__shfl_sync(kAll, qx.hi, k), __shfl_sync(kAll, qx.lo, k)};
          oy = F32Pair{__shfl_sync(kAll, qy.hi, k), __shfl_sync(kAll, qy.lo, k)};
        }
        V fax, fay;
        keep(ax, ay, ox, oy, fax, fay);
        V fbx = __shfl_up_sync(kAll, fax, 1), fby = __shfl_up_sync(kAll, fay, 1);
        if (lane == 0) {
          fbx = cx;
          fby = cy;
        }
        V const wx = __shfl_sync(kAll, zx, k), wy = __shfl_sync(kAll, zy, k);
        if ((beg >> lane) & 1u) {
          fbx = wx;
          fby = wy;
        }
        cx = __shfl_sync(kAll, fax, 31);
        cy = __shfl_sync(kAll, fay, 31);
        if constexpr (Filtered) {
          float const tx = __fmaf_rn(9.5367431640625e-07f, fmaxf(fabsf(fax), fabsf(fbx)),
                                     __fmaf_rn(4.547473508864641e-13f, fabsf(ox.hi),
                                               8.673617379884035e-19f));
          float const ty = __fmaf_rn(9.5367431640625e-07f, fmaxf(fabsf(fay), fabsf(fby)),
                                     __fmaf_rn(4.547473508864641e-13f, fabsf(oy.hi),
                                               8.673617379884035e-19f));
          if (own && fabsf(fay) > ty && fabsf(fby) > ty) {
            bool const y1 = fay > 0.0f, y0 = fby > 0.0f;
            if (y1 == y0) {
              und = !(fabsf(fax) > tx || fabsf(fbx) > tx);
            } else if (fabsf(fax) > tx && fabsf(fbx) > tx && (fax > 0.0f) == (fbx > 0.0f)) {
              tog = fax > 0.0f;
              und = false;
            } else {
              float const cr = __fmaf_rn(fay, fbx, -(fax * fby));
              float const eb = 2.0f * __fmaf_rn(tx, fabsf(fay) + fabsf(fby),
                                                ty * (fabsf(fax) + fabsf(fbx)));
              und            = !(fabsf(cr) > eb && fabsf(cr) < INFINITY);
              tog            = !und && (cr < 0.0f) != y1;
            }
          }
        }
        if (__any_sync(kAll, und)) {
          // the edge in the reference's arithmetic
          T bx, by, qpx, qpy;
          if constexpr (Filtered) {
            uint32_t const ek = __shfl_sync(kAll, e, k);
            uint32_t const pk = __shfl_sync(kAll, pl, k);
            uint32_t const sk = __shfl_sync(kAll, s, k);
            uint32_t const u  = v == sk ? ek - 1u : v - 1u;
            if (und) {
              bx  = vx[u];
              by  = vy[u];
              qpx = x[base + pk];
              qpy = y[base + pk];
            }
          } else {
            bx  = fbx;
            by  = fby;
            qpx = __shfl_sync(kAll, rpx, k);
            qpy = __shfl_sync(kAll, rpy, k);
          }
          if (und) {
            bool const ex = same_bits(ax, bx), ey = same_bits(ay, by);
            if (!(isfinite(ax) && isfinite(ay)) ||
                ((ex || (tiny_bits(ax) && tiny_bits(bx))) &&
                 (ey || (tiny_bits(ay) && tiny_bits(by))) && !(ex && ey))) {
              lit = true;  // the reference's skip rule needs the sequential walk
            } else if (!(ex && ey)) {  // a repeated vertex is skipped, b kept
              if (Filtered) ++nref;
              int const ee = exact_edge<T>(qpx, qpy, ax, ay, bx, by);
              hit          = ee == 2;
              tog          = ee == 1;
            }
          }
        }
        unsigned const bt = __ballot_sync(kAll, tog);
        unsigned const bh = __ballot_sync(kAll, hit);
        unsigned const bl = __ballot_sync(kAll, lit);
        if ((bt | bh | bl) != 0u) {
          // the lanes of ring j in this chunk
          uint32_t const lo   = s > c ? (s - c < 32u ? s - c : 32u) : 0u;
          uint32_t const hi   = e > c ? (e - c < 32u ? e - c : 32u) : 0u;
          unsigned const upto = hi ? kAll >> (32u - hi) : 0u;
          unsigned const from = lo < 32u ? kAll << lo : 0u;
          unsigned const mine = lane < nr ? upto & from : 0u;
          rpar                = rpar != static_cast<bool>(__popc(bt & mine) & 1u);
          ron |= (bh & mine) != 0u;
          rlit |= (bl & mine) != 0u;
        }
      }
      // rings [r0, r1) of pair p within this batch
      uint32_t const lo   = r0 > rr ? (r0 - rr < 32u ? r0 - rr : 32u) : 0u;
      uint32_t const hi   = r1 > rr ? (r1 - rr < 32u ? r1 - rr : 32u) : 0u;
      unsigned const upto = hi ? kAll >> (32u - hi) : 0u;
      unsigned const from = lo < 32u ? kAll << lo : 0u;
      unsigned const mine = upto & from;
      unsigned const bp   = __ballot_sync(kAll, rpar);
      unsigned const bo   = __ballot_sync(kAll, ron);
      unsigned const bq   = __ballot_sync(kAll, rlit);
      within              = within != static_cast<bool>(__popc(bp & mine) & 1u);
      on |= (bo & mine) != 0u;
      literal |= (bq & mine) != 0u;
    }
    if (have_p) {
      bool hit = !on && within;
      if (literal) {
        PolygonIndexView<T> v{};
        v.poly_offsets = po;
        v.ring_offsets = ro;
        v.vx           = vx;
        v.vy           = vy;
        hit            = ring_walk<T>(px, py, v, static_cast<uint32_t>(i));
      }
      out[i] = hit ? 1 : 0;
    }
  }
  if (Filtered && refined) {
    for (int o = 16; o > 0; o >>= 1) nref += __shfl_xor_sync(kAll, nref, o);
    if (lane == 0 && nref) atomicAdd(refined, static_cast<unsigned long long>(nref));
  }
}

// One lane per pair walks its polygon with the reference's loop.
template <typename T>
__global__ void __launch_bounds__(kPointsBlock)
  pairwise_lane_kernel(T const* __restrict__ x, T const* __restrict__ y, size_t n,
                       PolygonIndexView<T> v, uint8_t* __restrict__ out)
{
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[i] = ring_walk<T>(x[i], y[i], v, static_cast<uint32_t>(i)) ? 1 : 0;
}

unsigned points_grid(size_t n)
{
  return grid_for(n, kPointsBlock, static_cast<unsigned>(num_sms()) * 8u);
}

// log2 of the lanes per point: the smallest power of two >= the polygons
uint32_t lanes_log2(size_t npoly)
{
  uint32_t lp = 0;
  while ((size_t{1} << lp) < npoly) ++lp;
  return lp;
}

// Whether the bitmask call takes the grid of cells: where building it costs less
// than it saves.  31 polygons of 400 sides, 130k points, whole call: filtered
// 144 us with the grid, 155 without, exact 129 and 304; 65536 points of 1000
// sides: filtered 175 and 150, exact 157 and 229.  5 polygons of 20000 sides, 140k
// points: filtered 1251 and 888, exact 1224 and 1487 (2M points: 998 and 1402), so
// the filtered method asks for two points a vertex.
bool points_use_grid(size_t n, size_t nv, bool filtered)
{
  return filtered ? n >= (size_t{1} << 17) && n / 2 >= nv : n >= (size_t{1} << 16);
}
// The filtered method takes the grid where the median polygon's box is this many
// cells wide and high at least.  Cells that are large beside the polygons, or
// farther from the origin than float32 resolves them, decide little, and the tests
// they leave cost more than the filter's: 31 polygons of 100 sides in two places
// 10000 radii apart, 10M points around them: 23.7 ms with the grid, 7.2 without; one
// of 31 polygons of 1000 sides 100 radii off, 2M points around the others (5 cells a
// polygon): 1069 us and 639, 10M points (10 cells): 2536 and 2610.  (Where few
// polygons overlap fewer cells would do: 31 of 1000 sides spread over 20 radii, 140k
// points, 6 cells: 458 us and 1021.)  The exact method gains in all of these.
constexpr double kCellsPerPolygon = 8.0;

// Cells along an axis: one cell for every kPointsPerCell points.
uint32_t grid_side(size_t n)
{
  uint32_t g = kGridMin;
  while (g < kGridMax && static_cast<size_t>(g) * g * 4 * kPointsPerCell <= n) g *= 2;
  return g;
}

// Points 32 at a time a warp of the grid kernel takes together: as many as
// leave 32 warps for every SM.
uint32_t points_sets(size_t n)
{
  size_t const k = n / (static_cast<size_t>(num_sms()) * 32u * 32u);
  return static_cast<uint32_t>(k < 1 ? 1 : (k > kPointSets ? kPointSets : k));
}

void bitmask_grid(double const* x, double const* y, size_t n, PolygonIndex<double>& index,
                  size_t npoly, double bounds_share, Allocator const& alloc, int32_t* out,
                  unsigned long long* refined)
{
  cudaStream_t const s = alloc.stream();
  uint32_t const g = grid_side(n), sets = points_sets(n);
  Buffer<uint2> cells(alloc, static_cast<size_t>(g) * g);
  CSPT_CUDA_TRY(cudaMemsetAsync(cells.data(), 0, static_cast<size_t>(g) * g * sizeof(uint2), s));
  uint32_t const segs  = g * (g / 32u);
  uint32_t const share = std::max(1u, std::min(static_cast<uint32_t>(npoly), 32768u / segs));
  points_cells_kernel<<<grid_for(static_cast<size_t>(segs) * share * 32, kPointsBlock,
                                 sm_grid(8u)),
                        kPointsBlock, 0, s>>>(index.view(), bounds_share, g, share, cells.data());
  CSPT_CHECK_LAUNCH();
  points_grid_kernel<<<points_grid((n + sets - 1) / sets), kPointsBlock, 0, s>>>(
    x, y, n, index.view(), bounds_share, g, cells.data(), sets, out, refined);
  CSPT_CHECK_LAUNCH();
}

template <typename T>
void bitmask(T const* x, T const* y, size_t n, uint32_t const* po, size_t npo, uint32_t const* ro,
             size_t nro, T const* vx, T const* vy, size_t nv, bool filtered, Allocator const& alloc,
             int32_t* out, uint64_t* out_refined)
{
  cudaStream_t const s = alloc.stream();
  Buffer<unsigned long long> refined(alloc, 1);
  CSPT_CUDA_TRY(cudaMemsetAsync(refined.data(), 0, sizeof(unsigned long long), s));
  bool const grid =
    std::is_same<T, double>::value && points_use_grid(n, nv, filtered) && !alloc.frugal();
  // filtered: the device chooses by the polygons' sizes, and the kernels of the other
  // way return at once
  T const bounds_share = grid && filtered ? T{kCellsPerPolygon / grid_side(n)} : T{0};
  PolygonIndex<T> index(po, npo, ro, nro, vx, vy, nv, filtered, alloc, false, false, grid,
                        bounds_share);
  KernelTimer timer("points_pip", s);
  if constexpr (std::is_same<T, double>::value)
    if (grid)
      bitmask_grid(x, y, n, index, npo - 1, bounds_share, alloc, out, refined.data());
  uint32_t const lp = lanes_log2(npo - 1);
  if (filtered) {
    if constexpr (std::is_same<T, double>::value) {
      points_pip_kernel<double, true><<<points_grid(n), kPointsBlock, 0, s>>>(
        x, y, n, index.view(), bounds_share, lp, out, refined.data());
      CSPT_CHECK_LAUNCH();
    }
  } else if (!grid) {
    points_pip_kernel<T, false>
      <<<points_grid(n), kPointsBlock, 0, s>>>(x, y, n, index.view(), T{0}, lp, out, nullptr);
    CSPT_CHECK_LAUNCH();
  }
  *out_refined = filtered ? read_back(reinterpret_cast<uint64_t*>(refined.data()), s) : 0;
}

template <typename T>
void pairwise(T const* x, T const* y, size_t n, uint32_t const* po, uint32_t const* ro,
              T const* vx, T const* vy, size_t nv, bool filtered, Allocator const& alloc,
              uint8_t* out, uint64_t* out_refined)
{
  cudaStream_t const s = alloc.stream();
  Buffer<unsigned long long> refined(alloc, 1);
  CSPT_CUDA_TRY(cudaMemsetAsync(refined.data(), 0, sizeof(unsigned long long), s));
  // Pairs per warp: 32 where that leaves 48 warps for every SM, fewer for
  // short columns, so that their polygons still spread over the GPU.
  size_t const fill       = n / (static_cast<size_t>(num_sms()) * 48u);
  uint32_t const per_warp = static_cast<uint32_t>(fill < 1 ? 1 : (fill > 32 ? 32 : fill));
  unsigned const grd      = grid_for((n + per_warp - 1) / per_warp * 32, kPointsBlock, sm_grid(64u));
  // Exact polygons of a few vertices: a lane walks one in fewer instructions than a
  // run of 32 costs (1M pairs of 4..8 float32 vertices: 43 us a call against 64;
  // float64, 5 vertices: 10k pairs 43 us against 55, 1M 173 against 192).  Around 12
  // vertices the two meet; above, lanes wait for the largest polygon of their warp
  // and read it uncoalesced.  The filter's runs are faster from the start (1M pairs
  // of 5 vertices: 108 us).
  bool const lanes = !filtered && nv < 12 * n;
  {
    KernelTimer timer("pairwise_pip", s);
    if (lanes) {
      PolygonIndexView<T> v{};
      v.poly_offsets = po;
      v.ring_offsets = ro;
      v.vx           = vx;
      v.vy           = vy;
      pairwise_lane_kernel<T><<<points_grid(n), kPointsBlock, 0, s>>>(x, y, n, v, out);
    } else if (filtered) {
      if constexpr (std::is_same<T, double>::value)
        pairwise_pip_kernel<double, true>
          <<<grd, kPointsBlock, 0, s>>>(x, y, n, po, ro, vx, vy, per_warp, out, refined.data());
    } else {
      pairwise_pip_kernel<T, false>
        <<<grd, kPointsBlock, 0, s>>>(x, y, n, po, ro, vx, vy, per_warp, out, nullptr);
    }
    CSPT_CHECK_LAUNCH();
  }
  *out_refined = filtered ? read_back(reinterpret_cast<uint64_t*>(refined.data()), s) : 0;
}

}  // namespace

void point_in_polygon(void const* x, void const* y, size_t n, uint32_t const* po, size_t npo,
                      uint32_t const* ro, size_t nro, void const* vx, void const* vy, size_t nv,
                      cspt_dtype dtype, cspt_method method, Allocator const& alloc, int32_t* out,
                      uint64_t* out_refined)
{
  bool const filtered = method == CSPT_METHOD_FILTERED && dtype == CSPT_FLOAT64;
  if (dtype == CSPT_FLOAT64)
    bitmask<double>(static_cast<double const*>(x), static_cast<double const*>(y), n, po, npo, ro,
                    nro, static_cast<double const*>(vx), static_cast<double const*>(vy), nv,
                    filtered, alloc, out, out_refined);
  else
    bitmask<float>(static_cast<float const*>(x), static_cast<float const*>(y), n, po, npo, ro,
                   nro, static_cast<float const*>(vx), static_cast<float const*>(vy), nv, false,
                   alloc, out, out_refined);
}

void pairwise_point_in_polygon(void const* x, void const* y, size_t n, uint32_t const* po,
                               uint32_t const* ro, void const* vx, void const* vy, size_t nv,
                               cspt_dtype dtype, cspt_method method, Allocator const& alloc,
                               uint8_t* out, uint64_t* out_refined)
{
  bool const filtered = method == CSPT_METHOD_FILTERED && dtype == CSPT_FLOAT64;
  if (dtype == CSPT_FLOAT64)
    pairwise<double>(static_cast<double const*>(x), static_cast<double const*>(y), n, po, ro,
                     static_cast<double const*>(vx), static_cast<double const*>(vy), nv,
                     filtered, alloc, out, out_refined);
  else
    pairwise<float>(static_cast<float const*>(x), static_cast<float const*>(y), n, po, ro,
                    static_cast<float const*>(vx), static_cast<float const*>(vy), nv, false,
                    alloc, out, out_refined);
}

}  // namespace cspt
