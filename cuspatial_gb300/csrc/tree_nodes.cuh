// Quadtree nodes of all levels from sorted Morton keys, for one tree and for a
// forest of trees over consecutive ranges of positions.
//
// Reference: cpp/include/cuspatial/detail/index/construction/phase_1.cuh:60-381
// and phase_2.cuh:56-345.
#pragma once

#include "common.cuh"
#include "radix_sort.cuh"

namespace cspt {
namespace {  // one copy per translation unit

// ---------------------------------------------------------------------------
// Nodes of all levels in one pass over the sorted keys.
//
// A sorted position i that starts a node at level l0 (its start level) also
// starts one at every finer level, and a level-l node is kept iff its parent
// holds more than max_size points; counts shrink with the level, so the kept
// nodes starting at i are the levels l0..K of one interval.  Both ends follow
// from a few keys around i:
//   * the level-l node starting at i (l >= l0) holds more than m points iff
//     key[i + m] shares its level-l prefix, i.e. iff l <= c with c read off
//     the highest differing bit of key[i] ^ key[i + m];
//   * the parent of (i, l0), l0 > 0, starts before i; it holds more than m
//     points if key[i + m] shares its prefix (c >= l0 - 1) or key[i - m] does,
//     holds at most m if neither of two keys m + 1 apart around i does, and
//     otherwise its start is searched in the m positions before i.
// So K = min(d - 1, c + 1) where the deeper levels are kept, else l0, and a
// node (i, l) is internal iff l < K.  Nodes are output level by level in key
// order: counting them per (level, tile of positions) and scanning the counts
// level-major gives every node its output row, and the first child of an
// internal node (i, l) is node (i, l + 1), which is also the reference's
// child offset (level_1_size plus the scan of child counts).
//
// Bound: the key stream (4 bytes a position, the window reads hit L1) and, on
// small inputs, launches; this replaces a scan, a count, a scan and a
// compaction per level (61 launches at depth 5, 171 at depth 15).
// ---------------------------------------------------------------------------
constexpr int kNodeBlock     = 256;
constexpr int kNodeRounds    = 8;  // rounds of 32 positions per warp
constexpr int kNodeTile      = kNodeBlock * kNodeRounds;
constexpr int kNodeLevels    = 16;
static_assert(kNodeTile == kSortTile, "a forest's nodes are counted by its sort tiles");
constexpr uint8_t kNoNodes   = 0xFF;  // no kept node starts here (l0 and K are below 15)

// the deepest level at which two keys that differ in `diff` share their node,
// -1 if none
__device__ inline int shared_level(uint32_t diff, int d)
{
  if (diff == 0) return d - 1;
  int const c = d - 2 - (31 - __clz(diff)) / 2;
  return c < 0 ? -1 : c;
}

// l0 | K << 4 of position i of a tree over positions [b, n), kNoNodes when no
// kept node starts there
template <typename K>
__device__ inline uint8_t node_levels(K const* __restrict__ skeys, size_t b, size_t n, size_t i,
                                      int d, size_t m)
{
  K const key = skeys[i];
  int l0      = 0;
  if (i > b) {
    uint32_t const diff = static_cast<uint32_t>(key ^ skeys[i - 1]);
    if (diff == 0) return kNoNodes;
    l0 = d - 1 - (31 - __clz(diff)) / 2;
    l0 = l0 < 0 ? 0 : l0;
  }
  int const sh = 2 * (d - l0);  // the parent's prefix (l0 > 0: 2 <= sh < 32)
  K const P    = l0 > 0 ? key >> sh : K{0};
  if (l0 > 0) {
    // first the common case, a small parent: at most ha - 1 of its points lie
    // before i and hb from i on
    size_t const ha = (m + 1) / 2, hb = m + 1 - ha;
    if (!(i >= b + ha && (skeys[i - ha] >> sh) == P) && !(i + hb < n && (skeys[i + hb] >> sh) == P))
      return kNoNodes;
  }
  int const c = i + m < n ? shared_level(static_cast<uint32_t>(key ^ skeys[i + m]), d) : -1;
  if (c >= 0 && c >= l0 - 1) return static_cast<uint8_t>(l0 | (min(c + 1, d - 1) << 4));
  if (l0 > 0 && !(i >= b + m && (skeys[i - m] >> sh) == P)) {
    // the parent's first position, in (i - m, i - 1] (i - 1 belongs to it)
    size_t lo = i >= b + m ? i - m + 1 : b, hi = i - 1;
    while (lo < hi) {
      size_t const mid = (lo + hi) >> 1;
      if ((skeys[mid] >> sh) == P)
        hi = mid;
      else
        lo = mid + 1;
    }
    if (!(lo + m < n && (skeys[lo + m] >> sh) == P)) return kNoNodes;
  }
  return static_cast<uint8_t>(l0 | (l0 << 4));
}

// What a tile of positions belongs to: its positions [begin, end), its tree's
// positions [b, e), depth and leaf size, the row of the counts for each level and
// the tree's first node.
struct NodeTile {
  size_t begin, end, b, e;
  int d;
  size_t m;
  size_t row, step;  // level l at row + l step
  uint32_t base_row;  // its scanned count is the tree's first node
};
// one tree over positions [0, n)
struct OneTreeTiles {
  size_t n;
  unsigned ntiles;
  int d;
  size_t m;
  template <typename K>
  __device__ K mask() const  // the Morton bits of a key
  {
    return ~K{0};
  }
  template <typename K>
  __device__ NodeTile at(K const*, unsigned t) const
  {
    size_t const begin = static_cast<size_t>(t) * kNodeTile;
    return NodeTile{begin, begin + kNodeTile < n ? begin + kNodeTile : n, 0, n, d, m, t, ntiles, 0u};
  }
};

// The levels of a code as bits: a round of 32 positions holds nodes of few levels
// (node_write_kernel over all of them, 50M positions: 600 us, 236 this way).
__device__ inline unsigned level_bits(uint8_t code)
{
  return code == kNoNodes ? 0u : (2u << (code >> 4)) - (1u << (code & 15));
}

// Per position the levels of its kept nodes, per tile the nodes of each level
// (`levels` of them).  A forest's local point indices are written on the way;
// wide (null unless the sum may not fit 32 bits) receives the number of nodes.
template <typename K, typename Tiles>
__global__ void __launch_bounds__(kNodeBlock)
  node_count_kernel(K const* __restrict__ skeys, Tiles tiles, int levels,
                    uint8_t* __restrict__ codes, uint32_t* __restrict__ counts,
                    uint32_t const* __restrict__ sidx, uint32_t* __restrict__ local_idx,
                    unsigned long long* __restrict__ wide)
{
  __shared__ uint32_t cnt[kNodeLevels];
  if (threadIdx.x < kNodeLevels) cnt[threadIdx.x] = 0;
  __syncthreads();
  NodeTile const T = tiles.at(skeys, blockIdx.x);
#pragma unroll 2
  for (int r = 0; r < kNodeRounds; ++r) {
    size_t const i = T.begin + static_cast<size_t>(r) * kNodeBlock + threadIdx.x;
    if (i >= T.end) break;
    uint8_t const code = node_levels<K>(skeys, T.b, T.e, i, T.d, T.m);
    codes[i]           = code;
    if (local_idx) local_idx[i] = sidx[i] - static_cast<uint32_t>(T.b);
    if (code != kNoNodes)
      for (int l = code & 15; l <= (code >> 4); ++l) atomicAdd(&cnt[l], 1u);
  }
  __syncthreads();
  if (threadIdx.x < levels) {
    uint32_t const c                  = cnt[threadIdx.x];
    counts[T.row + threadIdx.x * T.step] = c;
    if (wide && c) atomicAdd(wide, static_cast<unsigned long long>(c));
  }
}

// The nodes' output columns; goff (may be null): a leaf's first position among
// all positions, 0 for internal nodes.  Offsets count from the tree's own
// first position and first node.
struct NodeColumns {
  uint32_t* key;
  uint8_t* level;
  uint8_t* internal;
  uint32_t* length;
  uint32_t* offset;
  uint32_t* goff;
};

// Writes the kept nodes of a tile at the rows that the scanned counts give.
// Warp w owns 256 consecutive positions; lane l keeps the running row of
// level l.  The child counts of internal nodes follow in child_count_kernel.
template <typename K, typename Tiles>
__global__ void __launch_bounds__(kNodeBlock)
  node_write_kernel(K const* __restrict__ skeys, Tiles tiles, uint8_t const* __restrict__ codes,
                    uint32_t const* __restrict__ rows, NodeColumns const out)
{
  constexpr unsigned kAll = 0xFFFFFFFFu;
  __shared__ uint32_t wcnt[kNodeBlock / 32][kNodeLevels];
  __shared__ uint32_t wfirst[kNodeBlock / 32];  // first position with nodes, in the tile
  int const lane    = threadIdx.x & 31;
  int const warp    = threadIdx.x >> 5;
  unsigned const lt = (1u << lane) - 1u;
  NodeTile const T   = tiles.at(skeys, blockIdx.x);
  int const d        = T.d;
  size_t const base  = T.begin + static_cast<size_t>(warp) * (32 * kNodeRounds);
  uint32_t const root = rows[T.base_row];  // the tree's first node
  uint8_t code[kNodeRounds];
#pragma unroll
  for (int r = 0; r < kNodeRounds; ++r) {
    size_t const i = base + r * 32 + lane;
    code[r]        = i < T.end ? codes[i] : kNoNodes;
  }
  uint32_t run   = 0;  // lane l: nodes of level l in this warp's positions
  uint32_t first = kNodeTile;
  unsigned starts[kNodeRounds];
#pragma unroll
  for (int r = kNodeRounds - 1; r >= 0; --r) {
    starts[r] = __ballot_sync(kAll, code[r] != kNoNodes);
    if (starts[r]) first = warp * (32 * kNodeRounds) + r * 32 + __ffs(starts[r]) - 1;
  }
#pragma unroll
  for (int r = 0; r < kNodeRounds; ++r) {
    if (!starts[r]) continue;
    unsigned const mine = level_bits(code[r]);
    for (unsigned ls = __reduce_or_sync(kAll, mine); ls; ls &= ls - 1u) {
      int const l      = __ffs(ls) - 1;
      unsigned const b = __ballot_sync(kAll, (mine >> l) & 1u);
      if (lane == l) run += __popc(b);
    }
  }
  if (lane < kNodeLevels) wcnt[warp][lane] = run;
  if (lane == 0) wfirst[warp] = first;
  __syncthreads();
  // the next position with nodes after this warp's, if it lies in the tile
  uint32_t after = kNodeTile;
  for (int w = kNodeBlock / 32 - 1; w > warp; --w)
    if (wfirst[w] < kNodeTile) after = wfirst[w];
  run = 0;
  if (lane < d) {
    run = rows[T.row + lane * T.step];
    for (int w = 0; w < warp; ++w) run += wcnt[w][lane];
  }
#pragma unroll
  for (int r = 0; r < kNodeRounds; ++r) {
    if (!starts[r]) continue;
    size_t const i     = base + r * 32 + lane;
    bool const any     = code[r] != kNoNodes;
    int const l0       = code[r] & 15, last = code[r] >> 4;
    K const key        = any ? skeys[i] : K{0};
    uint32_t parent    = 0;  // row of (i, l - 1)
    unsigned const levels = level_bits(code[r]);
    for (unsigned ls = __reduce_or_sync(kAll, levels); ls; ls &= ls - 1u) {
      int const l      = __ffs(ls) - 1;
      bool const mine  = (levels >> l) & 1u;
      unsigned const b = __ballot_sync(kAll, mine);
      uint32_t const o = __shfl_sync(kAll, run, l) + __popc(b & lt);
      if (lane == l) run += __popc(b);
      if (!mine) continue;
      out.key[o]      = static_cast<uint32_t>(key & tiles.template mask<K>()) >> (2 * (d - 1 - l));
      out.level[o]    = static_cast<uint8_t>(l);
      out.internal[o] = l < last ? 1 : 0;
      if (l > l0) {
        out.offset[parent] = o;  // made the tree's own in child_count_kernel
        if (out.goff) out.goff[parent] = root;
      }
      parent = o;
    }
    if (any) {
      // The leaf (i, last) ends where the next kept node starts: no kept node
      // starts inside a leaf, and the node after it is a sibling of it or of
      // one of its ancestors, which their parent's size keeps.  The tile's
      // last leaf looks for the first key beyond its prefix.
      uint32_t next = after;
#pragma unroll
      for (int t = kNodeRounds - 1; t >= r; --t) {
        unsigned const later = t == r ? starts[t] & ~lt & ~(1u << lane) : starts[t];
        if (later) next = warp * (32 * kNodeRounds) + t * 32 + __ffs(later) - 1;
      }
      size_t lo = T.begin + next;  // the end
      if (next == kNodeTile) {
        int const sh = 2 * (d - 1 - last);
        K const P    = key >> sh;
        size_t hi    = T.e;
        lo           = i + 1;  // the end lies in [lo, hi]
        for (size_t step = T.m; i + step < T.e; step *= 2) {
          if ((skeys[i + step] >> sh) != P) {
            hi = i + step;
            break;
          }
          lo = i + step + 1;
        }
        while (lo < hi) {
          size_t const mid = (lo + hi) >> 1;
          if ((skeys[mid] >> sh) == P)
            lo = mid + 1;
          else
            hi = mid;
        }
      }
      out.offset[parent] = static_cast<uint32_t>(i - T.b);
      out.length[parent] = static_cast<uint32_t>(lo - i);
      if (out.goff) out.goff[parent] = static_cast<uint32_t>(i);
    }
  }
}

// Children of an internal node: the rows from its first child on whose key
// extends the node's (at most four, all of the next level).  Its offset becomes
// the tree's own.
__global__ void child_count_kernel(NodeColumns const t, size_t q)
{
  for (size_t k = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; k < q;
       k += static_cast<size_t>(gridDim.x) * blockDim.x) {
    if (!t.internal[k]) continue;
    size_t const c0 = t.offset[k];
    uint32_t c      = 1;
    while (c < 4 && c0 + c < q && t.level[c0 + c] == t.level[c0] &&
           (t.key[c0 + c] >> 2) == t.key[k])
      ++c;
    t.length[k] = c;
    if (t.goff) {
      t.offset[k] -= t.goff[k];
      t.goff[k] = 0u;
    }
  }
}

template <typename K, typename Tiles>
void write_nodes(K const* skeys, Tiles const& tiles, unsigned ntiles, uint8_t const* codes,
                 uint32_t const* rows, NodeColumns const& out, size_t q, cudaStream_t s)
{
  node_write_kernel<K, Tiles><<<ntiles, kNodeBlock, 0, s>>>(skeys, tiles, codes, rows, out);
  CSPT_CHECK_LAUNCH();
  child_count_kernel<<<grid_for(q, 256, sm_grid(16u)), 256, 0, s>>>(out, q);
  CSPT_CHECK_LAUNCH();
}

// The rows are 32-bit: where up to `most` nodes might not fit, their number is
// summed in 64 bits and checked (one more wait), else nothing is allocated.
inline Buffer<unsigned long long> wide_node_total(size_t most, Allocator const& alloc)
{
  Buffer<unsigned long long> w(alloc, most >> 32 ? 1 : 0);
  if (w.data()) CSPT_CUDA_TRY(cudaMemsetAsync(w.data(), 0, sizeof(unsigned long long), alloc.stream()));
  return w;
}
inline void check_node_total(Buffer<unsigned long long> const& wide, cudaStream_t s)
{
  if (wide.data())
    CSPT_EXPECTS(read_back(wide.data(), s) < (1ull << 32), "the quadtree has 2^32 nodes or more");
}

}  // namespace
}  // namespace cspt
