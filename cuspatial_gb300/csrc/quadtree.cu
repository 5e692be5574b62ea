// Morton-key point quadtree on sm_103a.
//
// Reference: cpp/include/cuspatial/detail/point_quadtree.cuh:190-272 (clamps,
// construct_quadtree), detail/index/construction/phase_1.cuh:60-381 (keys,
// sort, bottom-up levels) and phase_2.cuh:56-345 (pruning, offsets).
//
// The reference builds every level bottom-up with reduce_by_key and then
// prunes.  Here the tree is read directly off the sorted keys, all levels in
// one pass (node_levels, tree_nodes.cuh): position i starts a node at level l exactly
// when the keys at i-1 and i differ in their level-l prefix, and a node at
// level l >= 1 is kept iff its parent holds more than max_size points, the
// reference's remove_unqualified_quads rule (phase_2.cuh:206-236).  Leaves
// keep the first sorted position they cover, which is what the reference's
// flattened-key scan (phase_2.cuh:98-141) produces.
#include <functional>
#include <limits>
#include <vector>

#include "common.cuh"
#include "radix_sort.cuh"
#include "scan.cuh"
#include "tree_nodes.cuh"

namespace cspt {
namespace {

constexpr uint8_t kNoStart = 0xFF;

// phase_1.cuh:73-85: out-of-box points take the last key of the deepest
// level; others interleave the truncated cell coordinates.
// Bound by the float64 pipe (two lanes a cycle and SM): a subtraction and a
// product per coordinate, and an fma near cell boundaries.  AtOrigin: the box
// starts at (0, 0) and v - 0 is v (50M points: 910 us, 533 this way; a whole tree
// of them 3860 us there, 4050 in a box elsewhere).  Four points a thread, all loads
// before the first key.
template <typename T, bool AtOrigin>
__global__ void __launch_bounds__(256)
  morton_keys_kernel(T const* __restrict__ x, T const* __restrict__ y, size_t n, T minx, T miny,
                     T maxx, T maxy, T scale, T rscale, int d, uint32_t* __restrict__ keys,
                     T* __restrict__ xy)
{
  constexpr int kPer = 4;
  size_t const step  = static_cast<size_t>(gridDim.x) * blockDim.x * kPer;
  for (size_t b = static_cast<size_t>(blockIdx.x) * blockDim.x * kPer + threadIdx.x; b < n;
       b += step) {
    T px[kPer], py[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      size_t const i = b + static_cast<size_t>(j) * blockDim.x;
      px[j]          = i < n ? x[i] : T{0};
      py[j]          = i < n ? y[i] : T{0};
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      size_t const i = b + static_cast<size_t>(j) * blockDim.x;
      if (i >= n) break;
      if (xy) {  // the points interleaved, in input order (for the ordered copy)
        if constexpr (sizeof(T) == 8)
          reinterpret_cast<double2*>(xy)[i] = make_double2(px[j], py[j]);
        else
          reinterpret_cast<float2*>(xy)[i] = make_float2(px[j], py[j]);
      }
      uint32_t k;
      if (outside_closed(px[j], minx, maxx) || outside_closed(py[j], miny, maxy)) {
        k = static_cast<uint32_t>((1 << (2 * d)) - 1);
      } else {
        uint16_t const cx = cell_of_quotient(AtOrigin ? px[j] : px[j] - minx, scale, rscale);
        uint16_t const cy = cell_of_quotient(AtOrigin ? py[j] : py[j] - miny, scale, rscale);
        k                 = (spread16(cy) << 1) | spread16(cx);
      }
      keys[i] = k;
    }
  }
}

__global__ void start_level_kernel(uint32_t const* __restrict__ skeys, size_t n, int d,
                                   uint8_t* __restrict__ lvl)
{
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    uint8_t l = 0;
    if (i > 0) {
      uint32_t const diff = skeys[i] ^ skeys[i - 1];
      if (diff == 0) {
        l = kNoStart;
      } else {
        int const h  = 31 - __clz(diff);
        int const lv = d - 1 - h / 2;
        l            = static_cast<uint8_t>(lv < 0 ? 0 : lv);
      }
    }
    lvl[i] = l;
  }
}

// sizes of the nodes of one level: count[k] = start[k+1] - start[k]
__global__ void bottom_count_kernel(uint32_t const* __restrict__ starts, size_t nl, size_t n,
                                  uint32_t* __restrict__ count)
{
  for (size_t k = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; k < nl;
       k += static_cast<size_t>(gridDim.x) * blockDim.x) {
    size_t const e = (k + 1 < nl) ? starts[k + 1] : n;
    count[k]       = static_cast<uint32_t>(e - starts[k]);
  }
}

// rows of an interleaved point array in quadtree order: dst[p] = src[pi[p]]
// (pi a permutation of [0, n)), four independent 16-byte (float64) or 8-byte
// (float32) gathers in flight per thread.
template <typename V>
__global__ void __launch_bounds__(256)
  gather_rows_kernel(uint32_t const* __restrict__ pi, size_t n, V const* __restrict__ src,
                     V* __restrict__ dst)
{
  constexpr int kPer = 4;
  size_t const step  = static_cast<size_t>(gridDim.x) * blockDim.x * kPer;
  for (size_t b = static_cast<size_t>(blockIdx.x) * blockDim.x * kPer + threadIdx.x; b < n;
       b += step) {
    uint32_t i[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      size_t const p = b + static_cast<size_t>(j) * blockDim.x;
      i[j]           = p < n ? pi[p] : 0u;
    }
    V v[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      size_t const p = b + static_cast<size_t>(j) * blockDim.x;
      if (p < n && i[j] < n) v[j] = src[i[j]];
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      size_t const p = b + static_cast<size_t>(j) * blockDim.x;
      if (p < n && i[j] < n) dst[p] = v[j];
    }
  }
}

// Host input: the points are copied from host memory (hx, hy) into the
// caller's device arrays (dx, dy, which build() then reads as x and y) in
// chunks on a second stream, and the Morton keys of each chunk are computed
// as soon as its copy has landed.  after_copies (may be null) is called with
// that stream once the points' copies are enqueued, so that a caller can
// queue more work behind them.
template <typename T>
struct HostInput {
  T const* hx;
  T const* hy;
  T* dx;
  T* dy;
  std::function<void(cudaStream_t)> const* after_copies;
};
// One chunk for every 4 Mi points (fewer leave a shorter merge: a host join of 20M
// points with 12 / 8 / 6 / 4 chunks 7734 / 7467 / 7378 / 7021 us), two from 2 Mi on,
// at most:
constexpr size_t kHostChunks = 8;

template <typename T>
void build(T const* x, T const* y, size_t n, double x1d, double x2d, double y1d, double y2d,
           double scaled, int max_depth_in, int32_t max_size_in, Allocator const& alloc,
           uint32_t** out_point_indices, cspt_quadtree* out, HostInput<T> const* host = nullptr,
           T* ordered = nullptr)
{
  cudaStream_t const s = alloc.stream();
  *out                 = cspt_quadtree{nullptr, nullptr, nullptr, nullptr, nullptr, 0};
  *out_point_indices   = nullptr;
  if (n == 0) return;
  CSPT_EXPECTS(n < (size_t{1} << 32), "quadtree_on_points supports fewer than 2^32 points");

  // detail/point_quadtree.cuh:258-268 — order the corners, clamp the
  // parameters (in the coordinate type, as the reference does).
  T const x1 = static_cast<T>(x1d), x2 = static_cast<T>(x2d);
  T const y1 = static_cast<T>(y1d), y2 = static_cast<T>(y2d);
  T const minx = x1 < x2 ? x1 : x2, maxx = x1 < x2 ? x2 : x1;
  T const miny = y1 < y2 ? y1 : y2, maxy = y1 < y2 ? y2 : y1;
  uint32_t const max_size = static_cast<uint32_t>(max_size_in < 1 ? 1 : max_size_in);
  int const d             = max_depth_in < 0 ? 0 : (max_depth_in > 15 ? 15 : max_depth_in);
  T const span            = (maxx - minx) > (maxy - miny) ? (maxx - minx) : (maxy - miny);
  T const min_scale       = span / static_cast<T>((1 << d) + 2);
  T scale                 = static_cast<T>(scaled);
  scale                   = scale > min_scale ? scale : min_scale;

  unsigned const blk = 256;
  unsigned const grd = grid_for(n, blk, sm_grid(16u));
  KernelTimer timer("quadtree_build", s);

  Buffer<uint32_t> keys(alloc, n), keys_alt(alloc, n);
  // (either may become the output, depending on the number of passes)
  Buffer<uint32_t> idx(alloc, n, OutputBuffer{}), idx_alt(alloc, n, OutputBuffer{});
  // ordered copy requested: the key pass also writes the points interleaved
  // (input order), so the gather after the sort reads one vector per point
  Buffer<T> xy_in(alloc, ordered ? 2 * n : 0);
  T* const xy0 = ordered ? xy_in.data() : nullptr;
  // cells reach 2^d + 2, so the key needs 2(d+1) bits (2(d+2) below d = 2)
  int const key_bits = d >= 2 ? 2 * d + 2 : 2 * d + 4;
  int const sort_bits = key_bits > 32 ? 32 : key_bits;
  bool alt = false;
  bool sorted = false;
  auto const morton_keys = [&](T const* px, T const* py, size_t m, uint32_t* out, T* interleaved) {
    unsigned const g = grid_for((m + 3) / 4, blk, sm_grid(16u));
    if (minx == T{0} && miny == T{0})
      morton_keys_kernel<T, true><<<g, blk, 0, s>>>(px, py, m, minx, miny, maxx, maxy, scale,
                                                    T{1} / scale, d, out, interleaved);
    else
      morton_keys_kernel<T, false><<<g, blk, 0, s>>>(px, py, m, minx, miny, maxx, maxy, scale,
                                                     T{1} / scale, d, out, interleaved);
    CSPT_CHECK_LAUNCH();
  };
  if (!host) {
    KernelTimer kt("quadtree_keys", s);
    morton_keys(x, y, n, keys.data(), xy0);
  } else {
    cudaStream_t const copy = side_stream();
    StreamJoin copies(s, copy);  // before `keys` is released, also on an exception
    stream_wait(copy, s);        // the destinations may come from work on s
    size_t const nch = std::min<size_t>(
      kHostChunks, std::max<size_t>(std::max<size_t>(1, n >> 22), std::min<size_t>(2, n >> 20)));
    // With several chunks each is sorted as soon as its keys exist, while
    // the next chunks are still crossing the link; the sorted chunks are
    // then merged (stable: equal keys keep their input order), which leaves
    // a short merge instead of the whole sort after the last copy.
    std::vector<size_t> runs{0};
    bool chunk_alt = false;
    for (size_t c = 0; c < nch; ++c) {
      size_t const i0 = n * c / nch, m = n * (c + 1) / nch - i0;
      CSPT_CUDA_TRY(cudaMemcpyAsync(host->dx + i0, host->hx + i0, m * sizeof(T),
                                    cudaMemcpyHostToDevice, copy));
      CSPT_CUDA_TRY(cudaMemcpyAsync(host->dy + i0, host->hy + i0, m * sizeof(T),
                                    cudaMemcpyHostToDevice, copy));
      stream_wait(s, copy);
      morton_keys(x + i0, y + i0, m, keys.data() + i0, xy0 ? xy0 + 2 * i0 : nullptr);
      if (nch > 1) {
        chunk_alt = radix_sort_pairs<uint32_t>(keys.data() + i0, idx.data() + i0,
                                               keys_alt.data() + i0, idx_alt.data() + i0, m, 0,
                                               sort_bits, true, alloc,
                                               static_cast<uint32_t>(i0));
        runs.push_back(i0 + m);
      }
    }
    if (host->after_copies) (*host->after_copies)(copy);
    copies.join();
    if (nch > 1) {
      KernelTimer kt("quadtree_sort", s);
      // every chunk took the same number of passes, so all runs sit in the
      // same pair of buffers
      bool const moved = chunk_alt ? merge_sorted_runs<uint32_t>(keys_alt.data(), idx_alt.data(),
                                                                keys.data(), idx.data(), runs, s)
                                   : merge_sorted_runs<uint32_t>(keys.data(), idx.data(),
                                                                keys_alt.data(), idx_alt.data(),
                                                                runs, s);
      alt    = chunk_alt != moved;
      sorted = true;
    }
  }
  if (!sorted) {
    KernelTimer kt("quadtree_sort", s);
    alt = radix_sort_pairs<uint32_t>(keys.data(), idx.data(), keys_alt.data(), idx_alt.data(), n,
                                     0, sort_bits, true, alloc);
  }
  Buffer<uint32_t>& skeys = alt ? keys_alt : keys;
  Buffer<uint32_t>& sidx  = alt ? idx_alt : idx;
  (alt ? keys : keys_alt).reset();
  // The ordered copy needs only the permutation: the gather (bound by
  // memory) runs on a second stream beside the levels (a chain of small
  // launches), and the caller's stream waits for it before the build returns
  // and before the interleaved input is released (order_join is destroyed
  // before xy_in, also on an exception).
  cudaStream_t const os = ordered ? side_stream() : nullptr;
  StreamJoin order_join(s, os);
  if (ordered) {
    stream_wait(os, s);  // the permutation and the interleaved input are on s
    KernelTimer kt("quadtree_order", os);
    unsigned const og = grid_for((n + 3) / 4, 256, sm_grid(8u));
    if constexpr (sizeof(T) == 8)
      gather_rows_kernel<double2><<<og, 256, 0, os>>>(
        sidx.data(), n, reinterpret_cast<double2 const*>(xy0), reinterpret_cast<double2*>(ordered));
    else
      gather_rows_kernel<float2><<<og, 256, 0, os>>>(
        sidx.data(), n, reinterpret_cast<float2 const*>(xy0), reinterpret_cast<float2*>(ordered));
    CSPT_CHECK_LAUNCH();
  }

  KernelTimer levels_timer("quadtree_levels", s);
  Buffer<uint32_t> total(alloc, 1);

  if (d <= 1) {
    // detail/point_quadtree.cuh:155-188: a tree of the bottom quadrants only
    Buffer<uint8_t> lvl(alloc, n);
    start_level_kernel<<<grd, blk, 0, s>>>(skeys.data(), n, d, lvl.data());
    CSPT_CHECK_LAUNCH();
    uint8_t const* lv = lvl.data();
    Buffer<uint32_t> starts(alloc, n);
    uint32_t* st = starts.data();
    scan_apply<uint32_t>(
      [lv] __device__(size_t i) { return lv[i] != kNoStart ? 1u : 0u; },
      [lv, st] __device__(size_t i, uint32_t e, uint32_t f) {
        if (f) st[e] = static_cast<uint32_t>(i);
      },
      n, total.data(), alloc);
    size_t const q = read_back(total.data(), s);
    OutputBuffer const out_tag;
    Buffer<uint32_t> okey(alloc, q, out_tag), olen(alloc, q, out_tag), ooff(alloc, q, out_tag);
    Buffer<uint8_t> olev(alloc, q, out_tag), oint(alloc, q, out_tag);
    bottom_count_kernel<<<grid_for(q, blk, sm_grid(16u)), blk, 0, s>>>(st, q, n, olen.data());
    CSPT_CHECK_LAUNCH();
    uint32_t const* sk = skeys.data();
    uint32_t* ok       = okey.data();
    uint32_t* oo       = ooff.data();
    scan_apply<uint32_t>([] __device__(size_t) { return 1u; },
                         [sk, st, ok, oo] __device__(size_t k, uint32_t, uint32_t) {
                           ok[k] = sk[st[k]];
                           oo[k] = st[k];
                         },
                         q, static_cast<uint32_t*>(nullptr), alloc);
    CSPT_CUDA_TRY(cudaMemsetAsync(olev.data(), 0, q, s));
    CSPT_CUDA_TRY(cudaMemsetAsync(oint.data(), 0, q, s));
    *out_point_indices = sidx.release();
    *out = cspt_quadtree{okey.release(), olev.release(), oint.release(), olen.release(),
                         ooff.release(), q};
    return;
  }

  // every level's nodes from one pass (node_levels); the host waits once, for
  // the number of nodes
  OneTreeTiles const tiles{n, static_cast<unsigned>((n + kNodeTile - 1) / kNodeTile), d, max_size};
  size_t const cells = static_cast<size_t>(tiles.ntiles) * d;
  Buffer<uint8_t> codes(alloc, n);
  Buffer<uint32_t> rows(alloc, cells);
  Buffer<unsigned long long> wide = wide_node_total(n * d, alloc);
  node_count_kernel<uint32_t, OneTreeTiles><<<tiles.ntiles, kNodeBlock, 0, s>>>(
    skeys.data(), tiles, d, codes.data(), rows.data(), nullptr, nullptr, wide.data());
  CSPT_CHECK_LAUNCH();
  check_node_total(wide, s);
  exclusive_scan<uint32_t>(rows.data(), rows.data(), cells, total.data(), alloc);
  size_t const q = read_back(total.data(), s);
  OutputBuffer const out_tag;
  Buffer<uint32_t> okey(alloc, q, out_tag), olen(alloc, q, out_tag), ooff(alloc, q, out_tag);
  Buffer<uint8_t> olev(alloc, q, out_tag), oint(alloc, q, out_tag);
  write_nodes<uint32_t>(skeys.data(), tiles, tiles.ntiles, codes.data(), rows.data(),
                        NodeColumns{okey.data(), olev.data(), oint.data(), olen.data(),
                                    ooff.data(), nullptr},
                        q, s);
  *out_point_indices = sidx.release();
  *out = cspt_quadtree{okey.release(), olev.release(), oint.release(), olen.release(),
                       ooff.release(), q};
}

// The points in quadtree order, interleaved: xy[pos] = (x[pi[pos]],
// y[pi[pos]]).  Each thread keeps four independent gathers in flight; the
// index reads and the 16-byte (float64) or 8-byte (float32) stores are
// coalesced.  An index at or beyond npts is never read through: its point
// becomes (NaN, NaN).
template <typename T, typename V>
__global__ void __launch_bounds__(256)
  ordered_points_kernel(uint32_t const* __restrict__ pi, size_t n, T const* __restrict__ x,
                        T const* __restrict__ y, size_t npts, V* __restrict__ xy)
{
  constexpr int kPer = 4;
  size_t const step  = static_cast<size_t>(gridDim.x) * blockDim.x * kPer;
  for (size_t b = static_cast<size_t>(blockIdx.x) * blockDim.x * kPer + threadIdx.x; b < n;
       b += step) {
    uint32_t i[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      size_t const p = b + static_cast<size_t>(j) * blockDim.x;
      i[j]           = p < n ? pi[p] : 0xFFFFFFFFu;
    }
    V v[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      bool const ok = i[j] < npts;
      v[j].x        = ok ? x[i[j]] : std::numeric_limits<T>::quiet_NaN();
      v[j].y        = ok ? y[i[j]] : std::numeric_limits<T>::quiet_NaN();
    }
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      size_t const p = b + static_cast<size_t>(j) * blockDim.x;
      if (p < n) xy[p] = v[j];
    }
  }
}

}  // namespace

void points_in_quadtree_order(uint32_t const* point_indices, size_t n, void const* x,
                              void const* y, size_t npts, cspt_dtype dtype, void* out_xy,
                              cudaStream_t s)
{
  if (n == 0) return;
  unsigned const grd = grid_for((n + 3) / 4, 256, sm_grid(8u));
  if (dtype == CSPT_FLOAT64)
    ordered_points_kernel<double, double2><<<grd, 256, 0, s>>>(
      point_indices, n, static_cast<double const*>(x), static_cast<double const*>(y), npts,
      static_cast<double2*>(out_xy));
  else
    ordered_points_kernel<float, float2><<<grd, 256, 0, s>>>(
      point_indices, n, static_cast<float const*>(x), static_cast<float const*>(y), npts,
      static_cast<float2*>(out_xy));
  CSPT_CHECK_LAUNCH();
}

void quadtree_on_points(void const* x, void const* y, size_t n, cspt_dtype dtype, double x_min,
                        double x_max, double y_min, double y_max, double scale, int max_depth,
                        int32_t max_size, Allocator const& alloc, uint32_t** out_point_indices,
                        cspt_quadtree* out_tree, void* ordered)
{
  if (dtype == CSPT_FLOAT64)
    build<double>(static_cast<double const*>(x), static_cast<double const*>(y), n, x_min, x_max,
                  y_min, y_max, scale, max_depth, max_size, alloc, out_point_indices, out_tree,
                  nullptr, static_cast<double*>(ordered));
  else
    build<float>(static_cast<float const*>(x), static_cast<float const*>(y), n, x_min, x_max,
                 y_min, y_max, scale, max_depth, max_size, alloc, out_point_indices, out_tree,
                 nullptr, static_cast<float*>(ordered));
}

void quadtree_on_points_from_host(void const* host_x, void const* host_y, void* dev_x,
                                  void* dev_y, size_t n, cspt_dtype dtype, double x_min,
                                  double x_max, double y_min, double y_max, double scale,
                                  int max_depth, int32_t max_size, Allocator const& alloc,
                                  uint32_t** out_point_indices, cspt_quadtree* out_tree,
                                  void* ordered,
                                  std::function<void(cudaStream_t)> const* after_copies)
{
  if (dtype == CSPT_FLOAT64) {
    HostInput<double> const h{static_cast<double const*>(host_x),
                              static_cast<double const*>(host_y), static_cast<double*>(dev_x),
                              static_cast<double*>(dev_y), after_copies};
    build<double>(h.dx, h.dy, n, x_min, x_max, y_min, y_max, scale, max_depth, max_size, alloc,
                  out_point_indices, out_tree, &h, static_cast<double*>(ordered));
  } else {
    HostInput<float> const h{static_cast<float const*>(host_x), static_cast<float const*>(host_y),
                             static_cast<float*>(dev_x), static_cast<float*>(dev_y),
                             after_copies};
    build<float>(h.dx, h.dy, n, x_min, x_max, y_min, y_max, scale, max_depth, max_size, alloc,
                 out_point_indices, out_tree, &h, static_cast<float*>(ordered));
  }
}

}  // namespace cspt
