// Quadrant / bounding-box intersection join on sm_103a.
//
// Reference: cpp/include/cuspatial/detail/join/quadtree_bbox_filtering.cuh:
// 35-188 (seeds, level loop, final stable sort by leaf offset),
// intersection.cuh:79-136 (node extent and closed-interval overlap) and
// traversal.cuh:57-145 (descent to children).
//
// The reference walks all boxes level by level with a host synchronisation
// per level.  Here a warp owns one box and walks the tree with a stack in
// shared memory (join_kernel.cuh).  The count pass sizes the output and
// appends every (node, box) it finds; a radix sort of the composite key
// (leaf first-point offset, box) gives the reference's order.  When the
// appended pairs would not fit, a write pass emits (leaf offset, box) in
// box-major order, a stable radix sort by the leaf offset gives the same order,
// and the nodes are looked up by their offsets.
// A node at traversal depth t is expanded only while t + 1 < max_depth, the
// reference's loop bound (quadtree_bbox_filtering.cuh:118).
#include <algorithm>
#include <cstddef>

#include "join_kernel.cuh"
#include "radix_sort.cuh"

namespace cspt {
namespace {

// Pairs the count pass may append (node + box, 8 bytes each): 64 per box, or, for
// few boxes over a large tree, all there can be up to 4 Mi; at most 64 Mi.  A join
// with more runs the write pass instead.  (frugal: 64 per box.)
inline size_t join_append_capacity(size_t nb, size_t nodes, bool frugal)
{
  size_t const all = frugal                             ? 0
                     : nodes < (size_t{4} << 20) / nb ? nodes * nb
                                                        : size_t{4} << 20;
  size_t const c   = std::max(nb * 64, all);
  return c < (size_t{64} << 20) ? c : (size_t{64} << 20);
}

// Warps per box: as many as give every SM 32 warps, with at least 256 nodes of the
// tree for each; the nodes four levels times as many are handed out.
inline JoinSplit join_split(size_t nb, size_t nodes, uint32_t* failed)
{
  JoinSplit p{1u, 0, failed};
  while (p.warps < 256u && nb * p.warps * 2 <= sm_grid(32u) && nodes >= p.warps * 512u)
    p.warps *= 2;
  while ((1u << (2 * p.level)) < 4u * p.warps) ++p.level;
  return p;
}

// (leaf first-point offset << box_bits) | box of each appended pair.
__global__ void composite_key_kernel(uint32_t const* __restrict__ node,
                                     uint32_t const* __restrict__ box, size_t k,
                                     uint32_t const* __restrict__ offset, int box_bits,
                                     uint64_t* __restrict__ key)
{
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < k;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    key[i] = (static_cast<uint64_t>(offset[node[i]]) << box_bits) | box[i];
}

// at[first point of a leaf] = the leaf's node + 1, over zeros; *shared is set where
// two leaves begin at the same point.
__global__ void leaf_at_kernel(TreeView t, uint32_t max_offset, uint32_t* __restrict__ at,
                               uint32_t* __restrict__ shared)
{
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < t.nq;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    uint32_t const o = t.offset[i];
    if (t.internal[i] || o > max_offset) continue;
    if (atomicExch(at + o, static_cast<uint32_t>(i) + 1u) != 0u) *shared = 1u;
  }
}

// Bound by the read of the sorted first points and the write of the nodes: equal
// first points stand together, so the table is read from the L1 cache.
__global__ void node_lookup_kernel(uint32_t const* __restrict__ first, size_t k,
                                   uint32_t const* __restrict__ at, uint32_t* __restrict__ node)
{
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < k;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    node[i] = at[first[i]] - 1u;
}

// What the count pass leaves for the host, read back in one copy.
struct JoinTotals {
  uint32_t max_offset;  // largest leaf first-point offset found
  int error;
  unsigned long long appended;
  uint32_t pairs;
  uint32_t level0;  // the tree's level-0 nodes
  uint32_t failed;  // a walk by several warps per box gave up
  uint32_t pad;
};

__global__ void count_level0_kernel(uint8_t const* __restrict__ level, size_t nq,
                                    uint32_t* __restrict__ out)
{
  uint32_t c = 0;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < nq;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    c += level[i] == 0 ? 1u : 0u;
  c = __reduce_add_sync(0xFFFFFFFFu, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

template <typename T>
void run(cspt_quadtree const* tree, T const* bminx, T const* bminy, T const* bmaxx,
         T const* bmaxy, size_t nb, T vminx, T vminy, T scale, int max_depth,
         Allocator const& alloc, uint32_t** out_box, uint32_t** out_node, size_t* out_n)
{
  cudaStream_t const s = alloc.stream();
  TreeView tv{tree->key, tree->level, tree->is_internal_node, tree->length, tree->offset,
              tree->num_nodes};
  Buffer<JoinTotals> totals(alloc, 1);
  JoinTotals* const tot = totals.data();
  CSPT_CUDA_TRY(cudaMemsetAsync(tot, 0, sizeof(JoinTotals), s));
  // seeds: the number of level-0 nodes (quadtree_bbox_filtering.cuh:53-56)
  count_level0_kernel<<<grid_for(tree->num_nodes, 256, sm_grid(4u)), 256, 0, s>>>(
    tree->level, tree->num_nodes, &tot->level0);
  CSPT_CHECK_LAUNCH();
  CSPT_EXPECTS(tree->num_nodes < (size_t{1} << 28), "quadtree has too many nodes");
  OneTree<T> const trees{&tot->level0, static_cast<uint32_t>(tree->num_nodes), vminx, vminy, scale,
                         max_depth};
  Buffer<uint32_t> counts(alloc, nb);
  int* const err     = &tot->error;
  unsigned const blk = kJoinWarps * 32;
  unsigned const grd = grid_for(nb * 32, blk, sm_grid(16u));
  // the count pass also appends each (node, box) it finds while they fit
  size_t const cap = join_append_capacity(nb, tree->num_nodes, alloc.frugal());
  Buffer<uint32_t> app_node(alloc, cap), app_box(alloc, cap);
  auto const count = [&](JoinSplit const& split) {
    KernelTimer timer("join_count", s);
    if (split.warps > 1u)
      CSPT_CUDA_TRY(cudaMemsetAsync(counts.data(), 0, nb * sizeof(uint32_t), s));
    unsigned const g = grid_for(nb * split.warps * 32, blk, sm_grid(16u));
    join_warp_kernel<T, false><<<g, blk, 0, s>>>(
      tv, trees, bminx, bminy, bmaxx, bmaxy, nb, counts.data(), &tot->max_offset, nullptr,
      nullptr, nullptr, nullptr, err,
      JoinAppend{app_node.data(), app_box.data(), &tot->appended, cap}, split);
    CSPT_CHECK_LAUNCH();
    exclusive_scan<uint32_t>(counts.data(), counts.data(), nb, &tot->pairs, alloc);
    return read_back(tot, s);
  };
  JoinTotals h = count(join_split(nb, tree->num_nodes, &tot->failed));
  if (h.failed && h.error == 0) {  // (only nodes of more than four children)
    CSPT_CUDA_TRY(cudaMemsetAsync(&tot->max_offset, 0, offsetof(JoinTotals, level0), s));
    h = count(JoinSplit{1u, 0, nullptr});
  }
  size_t const k     = h.pairs;
  CSPT_EXPECTS(h.error == 0,
               "quadtree is malformed: a node index or child count is out of range");
  *out_n = k;
  if (k == 0) return;
  int key_bits = 1;
  while (key_bits < 32 && (h.max_offset >> key_bits) != 0) ++key_bits;
  Buffer<uint32_t> ob(alloc, k, OutputBuffer{}), on(alloc, k, OutputBuffer{});
  if (h.appended == k && k <= cap) {
    // Every pair was appended (in no particular order): sort them by
    // (leaf offset, box), one composite key, which is the order the write
    // pass and a stable sort by leaf offset give.
    int box_bits = 1;
    while (box_bits < 32 && ((nb - 1) >> box_bits) != 0) ++box_bits;
    Buffer<uint64_t> key(alloc, k), key_alt(alloc, k);
    Buffer<uint32_t> perm(alloc, k), perm_alt(alloc, k);
    {
      KernelTimer timer("join_write", s);
      composite_key_kernel<<<grid_for(k, 256, sm_grid(16u)), 256, 0, s>>>(
        app_node.data(), app_box.data(), k, tv.offset, box_bits, key.data());
      CSPT_CHECK_LAUNCH();
    }
    bool const alt = radix_sort_pairs<uint64_t>(key.data(), perm.data(), key_alt.data(),
                                                perm_alt.data(), k, 0, key_bits + box_bits, true,
                                                alloc);
    gather_pairs_kernel<<<grid_for(k, 256, sm_grid(16u)), 256, 0, s>>>(
      alt ? perm_alt.data() : perm.data(), app_node.data(), app_box.data(), k, ob.data(),
      on.data());
    CSPT_CHECK_LAUNCH();
  } else {
    app_node.reset();
    app_box.reset();
    Buffer<uint32_t> key(alloc, k), key_alt(alloc, k);
    auto const write = [&](uint32_t* node, uint32_t* box) {
      KernelTimer timer("join_write", s);
      join_warp_kernel<T, true><<<grd, blk, 0, s>>>(tv, trees, bminx, bminy, bmaxx, bmaxy, nb,
                                                    nullptr, nullptr, counts.data(), key.data(),
                                                    node, box, err);
      CSPT_CHECK_LAUNCH();
    };
    // Where every leaf has its own first point (any tree of the quadtree build) the
    // boxes are sorted along with the first points and the nodes are looked up from
    // the sorted first points, next to one another, in place of a random gather of
    // both columns (0.52 ms for 43M pairs; a nearest-linestring call over 5M points and
    // 20k linestrings 10.95 -> 10.51 ms).  The table has an entry per point up to the
    // last leaf found; it is made for at most four entries per pair, so that its
    // clearing costs less than the gather.  With the table the write pass holds up to
    // nine words a pair, without it eight, as a call short of memory does.
    size_t const entries = static_cast<size_t>(h.max_offset) + 1;
    bool lookup          = entries <= 4 * k && !alloc.frugal();
    Buffer<uint32_t> at;
    if (lookup) {
      at = Buffer<uint32_t>(alloc, entries + 1);
      CSPT_CUDA_TRY(cudaMemsetAsync(at.data(), 0, (entries + 1) * sizeof(uint32_t), s));
      leaf_at_kernel<<<grid_for(tree->num_nodes, 256, sm_grid(8u)), 256, 0, s>>>(
        tv, h.max_offset, at.data(), at.data() + entries);
      CSPT_CHECK_LAUNCH();
      lookup = read_back(at.data() + entries, s) == 0;
    }
    if (lookup) {
      Buffer<uint32_t> ob_alt(alloc, k, OutputBuffer{});
      write(nullptr, ob.data());
      bool const alt = radix_sort_pairs<uint32_t>(key.data(), ob.data(), key_alt.data(),
                                                  ob_alt.data(), k, 0, key_bits, false, alloc);
      node_lookup_kernel<<<grid_for(k, 256, sm_grid(16u)), 256, 0, s>>>(
        alt ? key_alt.data() : key.data(), k, at.data(), on.data());
      CSPT_CHECK_LAUNCH();
      *out_box  = (alt ? ob_alt : ob).release();
      *out_node = on.release();
      return;
    }
    at.reset();
    Buffer<uint32_t> node(alloc, k), box(alloc, k), perm(alloc, k), perm_alt(alloc, k);
    write(node.data(), box.data());
    bool const alt = radix_sort_pairs<uint32_t>(key.data(), perm.data(), key_alt.data(),
                                                perm_alt.data(), k, 0, key_bits, true, alloc);
    gather_pairs_kernel<<<grid_for(k, 256, sm_grid(16u)), 256, 0, s>>>(
      alt ? perm_alt.data() : perm.data(), node.data(), box.data(), k, ob.data(), on.data());
    CSPT_CHECK_LAUNCH();
  }
  *out_box  = ob.release();
  *out_node = on.release();
}

}  // namespace

void join_quadtree_and_bounding_boxes(cspt_quadtree const* tree, void const* bminx,
                                      void const* bminy, void const* bmaxx, void const* bmaxy,
                                      size_t nb, cspt_dtype dtype, double x_min, double y_min,
                                      double scale, int max_depth, Allocator const& alloc,
                                      uint32_t** out_box, uint32_t** out_node, size_t* out_n)
{
  if (dtype == CSPT_FLOAT64)
    run<double>(tree, static_cast<double const*>(bminx), static_cast<double const*>(bminy),
                static_cast<double const*>(bmaxx), static_cast<double const*>(bmaxy), nb, x_min,
                y_min, scale, max_depth, alloc, out_box, out_node, out_n);
  else
    run<float>(tree, static_cast<float const*>(bminx), static_cast<float const*>(bminy),
               static_cast<float const*>(bmaxx), static_cast<float const*>(bmaxy), nb,
               static_cast<float>(x_min), static_cast<float>(y_min), static_cast<float>(scale),
               max_depth, alloc, out_box, out_node, out_n);
}

}  // namespace cspt
