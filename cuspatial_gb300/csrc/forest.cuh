// A forest of point quadtrees, one per instance, built in one pass.
//
// Instance i owns points [pt_begin_i, pt_end_i) of concatenated x/y columns
// and has its own quadtree_on_points parameters.  The forest holds the
// concatenation of the per-instance results:
//   * point_indices: instance i's sorted point order at [pt_begin_i,
//     pt_end_i), values local to the instance (pidx) and global (sidx);
//   * quadtree: instance i's nodes at [node_offsets_i, node_offsets_{i+1}),
//     child and point offsets local to the instance, plus goff = the leaf's
//     first position in the global sorted order.
// Each instance's part equals what quadtree_on_points returns for it alone
// (cpp/include/cuspatial/detail/point_quadtree.cuh:237-272).
//
// Points carry the composite key (instance << kb) | morton key and are
// sorted once, each instance's points within their own range (they are
// instance-major already, so a segmented radix sort of the Morton bits
// gives the composite order): instances stay contiguous and each instance's
// points take their own stable Morton order.  The nodes of all levels then come
// from one pass (tree_nodes.cuh) over tiles of positions that never cross an
// instance: the counts are laid out instance-major, level-major within the
// instance, so that one scan gives every node its output row.
#pragma once

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "join_kernel.cuh"
#include "radix_sort.cuh"
#include "scan.cuh"
#include "tree_nodes.cuh"

namespace cspt {
namespace {

constexpr unsigned kBlk     = 256;
inline unsigned grid_cap() { return sm_grid(16u); }

struct Inst {
  double minx, miny, maxx, maxy, scale, rscale;
  uint32_t d, max_size;
  uint32_t pt_begin, pt_end;
  uint32_t poly_begin, poly_end;
  uint32_t node_base, nq, L0;
};

// the instance whose [begin, next begin) holds v; begins has ni + 1 sorted
// entries and begins[0] <= v < begins[ni]
__device__ inline uint32_t find_instance(uint32_t const* __restrict__ begins, uint32_t ni,
                                         uint32_t v)
{
  uint32_t lo = 0, hi = ni;
  while (hi - lo > 1) {
    uint32_t const mid = (lo + hi) >> 1;
    if (begins[mid] <= v)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

#define CSPT_GRID_STRIDE(i, n)                                                           \
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < (n); \
       i += static_cast<size_t>(gridDim.x) * blockDim.x)

// Point positions in tiles of 2^kTileShift: tile_inst[t] = the instance of
// the tile's first position, tile_inst[ntiles] = ni - 1.  A position's
// instance then lies in [tile_inst[t], tile_inst[t + 1]], usually one entry.
constexpr int kTileShift = 10;
inline size_t position_tiles(size_t n) { return (n + (size_t{1} << kTileShift) - 1) >> kTileShift; }

__global__ void tile_instance_kernel(uint32_t const* __restrict__ begins, uint32_t ni, size_t ntiles,
                                     uint32_t* __restrict__ tile_inst)
{
  CSPT_GRID_STRIDE(t, ntiles + 1)
  {
    tile_inst[t] = t < ntiles ? find_instance(begins, ni, static_cast<uint32_t>(t << kTileShift))
                              : ni - 1u;
  }
}

// find_instance narrowed by the tile table
__device__ inline uint32_t instance_of(uint32_t const* __restrict__ begins,
                                       uint32_t const* __restrict__ tile_inst, uint32_t v)
{
  uint32_t const t = v >> kTileShift;
  uint32_t lo = tile_inst[t], hi = tile_inst[t + 1] + 1u;
  while (hi - lo > 1) {
    uint32_t const mid = (lo + hi) >> 1;
    if (begins[mid] <= v)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// phase_1.cuh:73-85 per instance, tagged with the instance
template <typename K>
__global__ void keys_kernel(double const* __restrict__ x, double const* __restrict__ y, size_t n,
                            uint32_t const* __restrict__ pt_begin,
                            uint32_t const* __restrict__ tile_inst,
                            Inst const* __restrict__ inst, int kb, K* __restrict__ keys)
{
  CSPT_GRID_STRIDE(i, n)
  {
    uint32_t const k = instance_of(pt_begin, tile_inst, static_cast<uint32_t>(i));
    Inst const& I    = inst[k];
    double const px = x[i], py = y[i];
    uint32_t key;
    if (outside_closed(px, I.minx, I.maxx) || outside_closed(py, I.miny, I.maxy)) {
      key = (1u << (2 * I.d)) - 1u;
    } else {
      uint16_t const cx = cell_of_quotient(px - I.minx, I.scale, I.rscale);
      uint16_t const cy = cell_of_quotient(py - I.miny, I.scale, I.rscale);
      key               = (spread16(cy) << 1) | spread16(cx);
    }
    keys[i] = (static_cast<K>(k) << kb) | key;
  }
}

// The tiles of a forest (its sort tiles; each lies in one instance).
struct ForestTiles {
  SortTile const* tiles;
  Inst const* inst;
  int kb;  // Morton bits
  template <typename K>
  __device__ K mask() const
  {
    return static_cast<K>((K{1} << kb) - 1u);
  }
  template <typename K>
  __device__ NodeTile at(K const* skeys, unsigned t) const
  {
    SortTile const T = tiles[t];
    Inst const& I    = inst[static_cast<uint32_t>(skeys[T.begin] >> kb)];
    size_t const row = static_cast<size_t>(T.first) * kNodeLevels;
    return NodeTile{T.begin,      T.end,   I.pt_begin, I.pt_end, static_cast<int>(I.d), I.max_size,
                    row + (t - T.first), T.count, static_cast<uint32_t>(row)};
  }
};

// Node ranges of the instances from the scanned counts (total = one past the
// last); seg_first[i] = the instance's first tile, seg_first[ni] = all tiles.
__global__ void layout_kernel(uint32_t const* __restrict__ seg_first,
                              uint32_t const* __restrict__ rows, uint32_t const* total, uint32_t ni,
                              Inst* __restrict__ inst, uint64_t* __restrict__ node_offsets,
                              int* __restrict__ error)
{
  uint32_t const all = *total, tiles = seg_first[ni];
  auto const first_node = [&](uint32_t i) {
    uint32_t const t = seg_first[i];
    return t < tiles ? rows[static_cast<size_t>(t) * kNodeLevels] : all;
  };
  CSPT_GRID_STRIDE(i, static_cast<size_t>(ni) + 1)
  {
    uint32_t const base = i < ni ? first_node(static_cast<uint32_t>(i)) : all;
    node_offsets[i]     = base;
    if (i == ni) continue;
    uint32_t const t = seg_first[i], count = seg_first[i + 1] - t;
    uint32_t const nq = first_node(static_cast<uint32_t>(i) + 1u) - base;
    inst[i].node_base = base;
    inst[i].nq        = nq;
    inst[i].L0 = count ? rows[static_cast<size_t>(t) * kNodeLevels + count] - base : 0u;
    if (nq >= (1u << 28)) atomicExch(error, 1);
  }
}

__global__ void row_offsets_kernel(uint32_t const* __restrict__ pair_begin,
                                   uint64_t const* __restrict__ pair_out, uint32_t ni,
                                   uint64_t* __restrict__ row_offsets)
{
  CSPT_GRID_STRIDE(i, static_cast<size_t>(ni) + 1) { row_offsets[i] = pair_out[pair_begin[i]]; }
}

// rows -> instance-local point positions (and polygon indices when the
// instances own polygon ranges)
__global__ void localize_kernel(uint32_t* __restrict__ op, uint32_t* __restrict__ oq, size_t m,
                                uint32_t const* __restrict__ pt_begin,
                                uint32_t const* __restrict__ tile_inst,
                                Inst const* __restrict__ inst, bool local_polygons)
{
  CSPT_GRID_STRIDE(j, m)
  {
    uint32_t const pos = oq[j];
    Inst const& I      = inst[instance_of(pt_begin, tile_inst, pos)];
    oq[j]              = pos - I.pt_begin;
    if (local_polygons) op[j] = op[j] - I.poly_begin;
  }
}


// the tree a box of instance `of(b)` walks
template <typename InstanceOf>
struct ForestTrees {
  InstanceOf of;
  Inst const* inst;
  __device__ BoxTree<double> operator()(size_t b) const
  {
    Inst const& I = inst[of(b)];
    return BoxTree<double>{I.node_base, I.nq,     I.L0,    I.pt_begin,
                           I.minx,      I.miny,   I.scale, static_cast<int>(I.d)};
  }
};

class Forest {
 public:
  explicit Forest(Allocator const& alloc) : alloc_(&alloc) {}

  // Validates the parameters (the reference's join checks,
  // quadtree_bbox_filtering.cu:100-106), applies the clamps of
  // detail/point_quadtree.cuh:258-268 and uploads the instance table.
  // poly_off (host, may be null) gives the instances' polygon ranges.
  void setup(size_t ni, uint64_t const* h_pt_off, cspt_instance_params const* params,
             uint64_t const* h_poly_off)
  {
    Allocator const& a   = *alloc_;
    cudaStream_t const s = a.stream();
    ni_                  = ni;
    n_                   = h_pt_off[ni];
    CSPT_EXPECTS(n_ < (size_t{1} << 32), "fewer than 2^32 points are supported");
    std::vector<Inst> hi(ni);
    std::vector<uint32_t> h_ptb(ni + 1), h_pob(ni + 1);
    dmax_ = 1;
    for (size_t i = 0; i < ni; ++i) {
      cspt_instance_params const& p = params[i];
      CSPT_EXPECTS(h_pt_off[i] <= h_pt_off[i + 1] &&
                     (!h_poly_off || h_poly_off[i] <= h_poly_off[i + 1]),
                   "instance offsets must be non-decreasing");
      CSPT_EXPECTS(p.scale > 0, "scale must be positive");
      CSPT_EXPECTS(p.x_min < p.x_max && p.y_min < p.y_max,
                   "invalid bounding box (x_min, x_max, y_min, y_max)");
      CSPT_EXPECTS(p.max_depth > 0 && p.max_depth < 16,
                   "maximum depth must be positive and less than 16");
      Inst& I           = hi[i];
      I.minx            = p.x_min;
      I.miny            = p.y_min;
      I.maxx            = p.x_max;
      I.maxy            = p.y_max;
      I.d               = static_cast<uint32_t>(p.max_depth);
      double const span = std::max(p.x_max - p.x_min, p.y_max - p.y_min);
      double const ms   = span / static_cast<double>((1 << p.max_depth) + 2);
      I.scale           = p.scale > ms ? p.scale : ms;
      I.rscale          = 1.0 / I.scale;
      I.max_size        = static_cast<uint32_t>(p.max_size < 1 ? 1 : p.max_size);
      I.pt_begin        = static_cast<uint32_t>(h_pt_off[i]);
      I.pt_end          = static_cast<uint32_t>(h_pt_off[i + 1]);
      I.poly_begin      = h_poly_off ? static_cast<uint32_t>(h_poly_off[i]) : 0u;
      I.poly_end        = h_poly_off ? static_cast<uint32_t>(h_poly_off[i + 1]) : 0u;
      I.node_base = I.nq = I.L0 = 0;
      h_ptb[i]                  = I.pt_begin;
      h_pob[i]                  = I.poly_begin;
      dmax_                     = std::max(dmax_, p.max_depth);
    }
    h_ptb[ni] = static_cast<uint32_t>(n_);
    h_pob[ni] = h_poly_off ? static_cast<uint32_t>(h_poly_off[ni]) : 0u;
    inst_       = Buffer<Inst>(a, ni);
    pt_begin_   = Buffer<uint32_t>(a, ni + 1);
    poly_begin_ = Buffer<uint32_t>(a, ni + 1);
    CSPT_CUDA_TRY(cudaMemcpyAsync(inst_.data(), hi.data(), ni * sizeof(Inst),
                                  cudaMemcpyHostToDevice, s));
    CSPT_CUDA_TRY(cudaMemcpyAsync(pt_begin_.data(), h_ptb.data(), (ni + 1) * 4,
                                  cudaMemcpyHostToDevice, s));
    CSPT_CUDA_TRY(cudaMemcpyAsync(poly_begin_.data(), h_pob.data(), (ni + 1) * 4,
                                  cudaMemcpyHostToDevice, s));
    // radix sort tiles within instances: the points are instance-major
    // already, so only the Morton bits are sorted
    std::vector<uint64_t> bounds{0};
    for (size_t i = 1; i < ni; ++i) bounds.push_back(h_pt_off[i]);
    bounds.push_back(n_);
    std::vector<SortTile> hs;
    segment_sort_tiles(bounds, hs);
    sort_tiles_ = Buffer<SortTile>(a, hs.size());
    std::vector<uint32_t> hf(ni + 1);  // each instance's first tile
    for (size_t i = 0, t = 0; i < ni; ++i) {
      hf[i] = static_cast<uint32_t>(t);
      t += (h_pt_off[i + 1] - h_pt_off[i] + kSortTile - 1) / kSortTile;
      hf[i + 1] = static_cast<uint32_t>(t);
    }
    seg_first_ = Buffer<uint32_t>(a, ni + 1);
    CSPT_CUDA_TRY(cudaMemcpyAsync(seg_first_.data(), hf.data(), (ni + 1) * 4,
                                  cudaMemcpyHostToDevice, s));
    if (!hs.empty())
      CSPT_CUDA_TRY(cudaMemcpyAsync(sort_tiles_.data(), hs.data(), hs.size() * sizeof(SortTile),
                                    cudaMemcpyHostToDevice, s));
    size_t const ntiles = position_tiles(n_);
    tile_inst_          = Buffer<uint32_t>(a, ntiles + 1);
    if (ni) {
      tile_instance_kernel<<<grid_for(ntiles + 1, kBlk, grid_cap()), kBlk, 0, s>>>(
        pt_begin_.data(), static_cast<uint32_t>(ni), ntiles, tile_inst_.data());
      CSPT_CHECK_LAUNCH();
    }
    // the host arrays above must outlive the copies
    CSPT_CUDA_TRY(cudaStreamSynchronize(s));
  }

  void build(double const* x, double const* y)
  {
    Allocator const& a   = *alloc_;
    cudaStream_t const s = a.stream();
    size_t const n       = n_;
    node_off_            = Buffer<uint64_t>(a, ni_ + 1, OutputBuffer{});
    if (n == 0) {
      CSPT_CUDA_TRY(cudaMemsetAsync(node_off_.data(), 0, (ni_ + 1) * 8, s));
      return;
    }
    KernelTimer timer("forest_build", s);
    int const kb = dmax_ >= 2 ? 2 * dmax_ + 2 : 2 * dmax_ + 4;
    int ib       = 0;
    while ((uint64_t{1} << ib) < ni_) ++ib;
    // 32-bit composite keys when the instance and Morton bits fit: a third
    // less traffic in every sort pass
    if (kb + ib < 32)
      build_sorted<uint32_t>(x, y, kb);
    else
      build_sorted<uint64_t>(x, y, kb);
  }

  template <typename K>
  void build_sorted(double const* x, double const* y, int kb)
  {
    Allocator const& a   = *alloc_;
    cudaStream_t const s = a.stream();
    uint32_t const ni    = static_cast<uint32_t>(ni_);
    size_t const n       = n_;
    unsigned const grd   = grid_for(n, kBlk, grid_cap());

    Buffer<K> keys(a, n), keys_alt(a, n);
    Buffer<uint32_t> idx(a, n), idx_alt(a, n);
    keys_kernel<K><<<grd, kBlk, 0, s>>>(x, y, n, pt_begin_.data(), tile_inst_.data(), inst_.data(),
                                        kb, keys.data());
    CSPT_CHECK_LAUNCH();
    bool const alt = radix_sort_segments<K>(keys.data(), idx.data(), keys_alt.data(),
                                            idx_alt.data(), n, 0, kb, true, sort_tiles_.data(),
                                            static_cast<unsigned>(sort_tiles_.size()), a);
    Buffer<K>& sk = alt ? keys_alt : keys;
    sidx_         = std::move(alt ? idx_alt : idx);
    (alt ? keys : keys_alt).reset();
    (alt ? idx : idx_alt).reset();

    unsigned const ntiles = static_cast<unsigned>(sort_tiles_.size());
    ForestTiles const tiles{sort_tiles_.data(), inst_.data(), kb};
    size_t const cells = static_cast<size_t>(ntiles) * kNodeLevels;
    pidx_              = Buffer<uint32_t>(a, n, OutputBuffer{});
    Buffer<uint8_t> codes(a, n);
    Buffer<uint32_t> rows(a, cells), total(a, 2);  // nodes, error flag
    CSPT_CUDA_TRY(cudaMemsetAsync(total.data(), 0, 2 * sizeof(uint32_t), s));
    Buffer<unsigned long long> wide = wide_node_total(n * static_cast<size_t>(dmax_), a);
    node_count_kernel<K, ForestTiles><<<ntiles, kNodeBlock, 0, s>>>(
      sk.data(), tiles, kNodeLevels, codes.data(), rows.data(), sidx_.data(), pidx_.data(),
      wide.data());
    CSPT_CHECK_LAUNCH();
    static char const* const kTooMany =
      "an instance's quadtree has too many nodes for the batched form";
    if (wide.data()) CSPT_EXPECTS(read_back(wide.data(), s) < (1ull << 32), kTooMany);
    exclusive_scan<uint32_t>(rows.data(), rows.data(), cells, total.data(), a);
    layout_kernel<<<grid_for(ni_ + 1, kBlk, grid_cap()), kBlk, 0, s>>>(
      seg_first_.data(), rows.data(), total.data(), ni, inst_.data(), node_off_.data(),
      reinterpret_cast<int*>(total.data() + 1));
    CSPT_CHECK_LAUNCH();
    uint32_t h[2];
    CSPT_CUDA_TRY(cudaMemcpyAsync(h, total.data(), sizeof(h), cudaMemcpyDeviceToHost, s));
    CSPT_CUDA_TRY(cudaStreamSynchronize(s));
    CSPT_EXPECTS(h[1] == 0, kTooMany);
    size_t const q = q_ = h[0];
    OutputBuffer const out_tag;
    key_      = Buffer<uint32_t>(a, q, out_tag);
    length_   = Buffer<uint32_t>(a, q, out_tag);
    offset_   = Buffer<uint32_t>(a, q, out_tag);
    goff_     = Buffer<uint32_t>(a, q);
    level_    = Buffer<uint8_t>(a, q, out_tag);
    internal_ = Buffer<uint8_t>(a, q, out_tag);
    write_nodes<K>(sk.data(), tiles, ntiles, codes.data(), rows.data(),
                   NodeColumns{key_.data(), level_.data(), internal_.data(), length_.data(),
                               offset_.data(), goff_.data()},
                   q, s);
  }

  TreeView view() const
  {
    return TreeView{key_.data(), level_.data(), internal_.data(), length_.data(), offset_.data(),
                    q_};
  }
  cspt_quadtree tree() const
  {
    return cspt_quadtree{key_.data(), level_.data(), internal_.data(), length_.data(),
                         offset_.data(), q_};
  }

  Allocator const* alloc_;
  size_t ni_ = 0, n_ = 0, q_ = 0;
  int dmax_  = 1;
  Buffer<Inst> inst_;
  Buffer<uint32_t> pt_begin_, poly_begin_, tile_inst_, seg_first_;
  Buffer<SortTile> sort_tiles_;
  Buffer<uint32_t> sidx_, pidx_;
  Buffer<uint32_t> key_, length_, offset_, goff_;
  Buffer<uint8_t> level_, internal_;
  Buffer<uint64_t> node_off_;
};

}  // namespace
}  // namespace cspt
