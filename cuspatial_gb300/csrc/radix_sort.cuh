// Stable LSD radix sort of (key, uint32 value) pairs, 8-bit digits over a bit
// range, so Morton keys of depth d cost ceil(2(d+1)/8) passes instead of 4.
//
// Per pass: per-tile digit histograms -> exclusive scan in digit-major order
// -> stable scatter.  Within a tile each warp ranks its 256 consecutive items
// with __match_any_sync; tiles, warps, rounds and lanes follow input order,
// which keeps the sort stable.  A segmented form sorts each of many
// contiguous segments in place (tiles never cross a segment boundary).
#pragma once

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "scan.cuh"

namespace cspt {

constexpr int kSortBlock = 256;  // one thread per 8-bit digit in the scatter
constexpr int kSortWarps = kSortBlock / 32;
// Rounds of 32 items per warp.  A fixed constant, not a build option: the
// sort's templates are instantiated in several translation units, and one
// program must see one tile size in all of them.
constexpr int kSortRound = 8;
constexpr int kSortTile  = kSortBlock * kSortRound;
constexpr unsigned kNoDigit = 0xFFFFu;
constexpr uint32_t kNoItem  = 0xFFFFFFFFu;

// Where a tile's items lie and where its digit counts go.
// PlainTiles: fixed tiles over [0, n); counts digit-major over all tiles, so
// one exclusive scan of the counts gives each (digit, tile) its output start.
struct PlainTiles {
  size_t n;
  unsigned ntiles;
  __device__ void range(unsigned t, size_t& b, size_t& e) const
  {
    b = static_cast<size_t>(t) * kSortTile;
    e = b + kSortTile < n ? b + kSortTile : n;
  }
  __device__ size_t slot(unsigned t, unsigned d) const
  {
    return static_cast<size_t>(d) * ntiles + t;
  }
};
// SegmentTiles: tiles that never cross a segment boundary; counts
// segment-major, then digit-major within the segment.  One exclusive scan
// then sorts every segment within its own range: segments stay in place, so
// keys already ordered by their high bits per segment need only their low
// bits sorted.
struct SortTile {
  uint32_t begin, end;   // items [begin, end)
  uint32_t first, count; // the segment's first tile and its number of tiles
};
struct SegmentTiles {
  SortTile const* tiles;
  __device__ void range(unsigned t, size_t& b, size_t& e) const
  {
    b = tiles[t].begin;
    e = tiles[t].end;
  }
  __device__ size_t slot(unsigned t, unsigned d) const
  {
    SortTile const& T = tiles[t];
    return static_cast<size_t>(T.first) * 256 + static_cast<size_t>(d) * T.count + (t - T.first);
  }
};

// Digit counts of the tiles.  A block takes tile after tile, the next tile's keys
// loading while this one's are counted: one tile a block left the kernel waiting
// for its loads (50M keys: 116 us a pass, 59 this way).
template <typename K, typename Tiles>
__global__ void __launch_bounds__(kSortBlock)
  radix_histogram_kernel(K const* keys, Tiles tiles, unsigned ntiles, int shift, unsigned mask,
                         uint32_t* counts)
{
  __shared__ uint32_t hist[kSortWarps][256];
  int const warp = threadIdx.x >> 5;
  int const lane = threadIdx.x & 31;
  K key[kSortRound];
  unsigned valid = 0;  // rounds with a key
  auto const load = [&](unsigned t) {
    size_t tb, te;
    tiles.range(t, tb, te);
    size_t const base = tb + warp * (32 * kSortRound) + lane;
    valid             = 0;
#pragma unroll
    for (int r = 0; r < kSortRound; ++r) {
      bool const ok = base + r * 32 < te;
      key[r]        = ok ? keys[base + r * 32] : K{0};
      valid |= ok ? 1u << r : 0u;
    }
  };
  if (blockIdx.x < ntiles) load(blockIdx.x);
  for (unsigned t = blockIdx.x; t < ntiles; t += gridDim.x) {
    for (int i = threadIdx.x; i < kSortWarps * 256; i += kSortBlock) (&hist[0][0])[i] = 0;
    unsigned d[kSortRound];
    unsigned const own = valid;
#pragma unroll
    for (int r = 0; r < kSortRound; ++r) d[r] = static_cast<unsigned>((key[r] >> shift) & mask);
    if (t + gridDim.x < ntiles) load(t + gridDim.x);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortRound; ++r)
      if ((own >> r) & 1u) atomicAdd(&hist[warp][d[r]], 1u);
    __syncthreads();
    uint32_t s = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) s += hist[w][threadIdx.x];
    counts[tiles.slot(t, threadIdx.x)] = s;
    __syncthreads();
  }
}

static_assert(kSortBlock == 256, "the scatter assigns one thread per digit");

// Stable scatter of one tile: items are ranked per warp with
// __match_any_sync (rounds in input order), placed in shared memory in the
// tile's digit order, then written out in that order, so the global writes
// of each digit's run are contiguous.  Bound by its waits for shared memory (17 of
// them per issued instruction, the pipe 45% busy; 20M keys) and too few blocks to
// cover them: 50M pairs, four passes: 1657 us with keys and values apart and 61
// registers (four blocks an SM), 1423 us as here with six.
template <typename K, typename Tiles>
__global__ void __launch_bounds__(kSortBlock, 6)
  radix_scatter_kernel(K const* keys_in, uint32_t const* vals_in, K* keys_out, uint32_t* vals_out,
                       Tiles tiles, int shift, unsigned mask, uint32_t const* offsets,
                       uint32_t iota_base)
{
  __shared__ uint32_t wcount[kSortWarps][256];
  __shared__ uint32_t global_base[256];  // the digit's output start minus its tile start
  // (32-bit keys beside their values: one 64-bit access for both)
  constexpr bool kPacked = sizeof(K) == 4;
  __shared__ K skey[kPacked ? 1 : kSortTile];
  __shared__ uint32_t sval[kPacked ? 1 : kSortTile];
  __shared__ uint2 spair[kPacked ? kSortTile : 1];
  __shared__ uint32_t total_s;
  for (int i = threadIdx.x; i < kSortWarps * 256; i += kSortBlock) (&wcount[0][0])[i] = 0;
  __syncthreads();
  int const warp       = threadIdx.x >> 5;
  int const lane       = threadIdx.x & 31;
  unsigned const lt    = (1u << lane) - 1u;
  size_t tb, te;
  tiles.range(blockIdx.x, tb, te);
  size_t const base    = tb + warp * (32 * kSortRound);
  K key[kSortRound];
  uint32_t val[kSortRound];
  uint32_t meta[kSortRound];  // digit | rank in the warp's digit << 8, kNoItem
#pragma unroll
  for (int r = 0; r < kSortRound; ++r) {
    size_t const i = base + r * 32 + lane;
    bool const ok  = i < te;
    key[r]         = ok ? keys_in[i] : K{0};
    val[r]         = ok ? (vals_in ? vals_in[i] : static_cast<uint32_t>(i) + iota_base) : 0u;
    unsigned const dig   = ok ? static_cast<unsigned>((key[r] >> shift) & mask) : kNoDigit;
    unsigned const peers = __match_any_sync(0xFFFFFFFFu, dig);
    unsigned const below = __popc(peers & lt);
    uint32_t prior       = 0;
    if (ok) prior = wcount[warp][dig];
    meta[r] = ok ? dig | ((prior + below) << 8) : kNoItem;
    __syncwarp();
    // the lowest lane of each digit group advances the warp's counter
    if (ok && below == 0) wcount[warp][dig] = prior + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // per digit (one thread each): prefix over warps, the tile's digit start
  // and the digit's global base
  {
    int const d    = threadIdx.x;  // kSortBlock == 256 digits
    uint32_t run   = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) run += wcount[w][d];
    uint32_t at = block_exclusive_scan<uint32_t, kSortBlock>(run, &total_s);
    global_base[d] = offsets[tiles.slot(blockIdx.x, d)] - at;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {  // where the warp's items of the digit go
      uint32_t const c = wcount[w][d];
      wcount[w][d]     = at;
      at += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortRound; ++r) {
    if (meta[r] != kNoItem) {
      uint32_t const t = wcount[warp][meta[r] & 255u] + (meta[r] >> 8);
      if constexpr (kPacked) {
        spair[t] = make_uint2(static_cast<uint32_t>(key[r]), val[r]);
      } else {
        skey[t] = key[r];
        sval[t] = val[r];
      }
    }
  }
  __syncthreads();
  uint32_t const m = total_s;
  for (uint32_t t = threadIdx.x; t < m; t += kSortBlock) {
    K k;
    uint32_t v;
    if constexpr (kPacked) {
      uint2 const p = spair[t];
      k             = p.x;
      v             = p.y;
    } else {
      k = skey[t];
      v = sval[t];
    }
    uint32_t const g = global_base[static_cast<unsigned>((k >> shift) & mask)] + t;
    keys_out[g]      = k;
    vals_out[g]      = v;
  }
}

// Sorts (keys, vals) by bits [begin_bit, end_bit) of the key.  When
// iota_vals is set the incoming contents of vals are ignored and vals[i] =
// iota_base + i is used instead.  The result lands in (keys, vals) or in (keys_alt,
// vals_alt); the return value is true when it is in the _alt buffers.
// n must be below 2^32.
template <typename K, typename Tiles>
bool radix_sort_tiles(K* keys, uint32_t* vals, K* keys_alt, uint32_t* vals_alt, size_t n,
                      int begin_bit, int end_bit, bool iota_vals, Tiles tiles, unsigned ntiles,
                      Allocator const& alloc, uint32_t iota_base = 0)
{
  cudaStream_t const s = alloc.stream();
  if (n == 0) return false;
  if (end_bit <= begin_bit) {
    if (iota_vals) {
      scan_apply<uint32_t>(
        [] __device__(size_t) { return 1u; },
        [vals, iota_base] __device__(size_t i, uint32_t e, uint32_t) { vals[i] = e + iota_base; },
        n, static_cast<uint32_t*>(nullptr), alloc);
    }
    return false;
  }
  Buffer<uint32_t> counts(alloc, static_cast<size_t>(ntiles) * 256);
  bool in_alt = false;
  bool first  = true;
  for (int shift = begin_bit; shift < end_bit; shift += 8) {
    K* kin         = in_alt ? keys_alt : keys;
    uint32_t* vin  = in_alt ? vals_alt : vals;
    K* kout        = in_alt ? keys : keys_alt;
    uint32_t* vout = in_alt ? vals : vals_alt;
    int const width     = end_bit - shift < 8 ? end_bit - shift : 8;
    unsigned const mask = (1u << width) - 1u;
    radix_histogram_kernel<K, Tiles>
      <<<std::min(ntiles, sm_grid(8u)), kSortBlock, 0, s>>>(kin, tiles, ntiles, shift, mask,
                                                            counts.data());
    CSPT_CHECK_LAUNCH();
    exclusive_scan<uint32_t>(counts.data(), counts.data(), static_cast<size_t>(ntiles) * 256,
                             static_cast<uint32_t*>(nullptr), alloc);
    radix_scatter_kernel<K, Tiles><<<ntiles, kSortBlock, 0, s>>>(
      kin, (first && iota_vals) ? nullptr : vin, kout, vout, tiles, shift, mask, counts.data(),
      iota_base);
    CSPT_CHECK_LAUNCH();
    in_alt = !in_alt;
    first  = false;
  }
  return in_alt;
}

// One block sorts up to kSmallSort pairs: each pair's digits and its position
// make one 64-bit word, the words are unique, so a bitonic network (unstable)
// gives the stable order.  A radix pass is three launches and a call of the
// allocator whatever the size: 1003 Morton keys of 12 bits took 7 launches, now
// one.
constexpr unsigned kSmallSort     = 2048;
constexpr int kSmallPositionBits  = 11;
constexpr unsigned kSmallBlock    = kSmallSort / 2;

template <typename K>
__global__ void __launch_bounds__(kSmallBlock)
  small_sort_kernel(K* __restrict__ keys, uint32_t* __restrict__ vals, unsigned n, int begin_bit,
                    K mask, bool iota_vals, uint32_t iota_base)
{
  __shared__ unsigned long long word[kSmallSort];
  unsigned m = 2;  // a power of two, at least n
  while (m < n) m *= 2;
  for (unsigned i = threadIdx.x; i < m; i += kSmallBlock)
    word[i] = i < n ? (static_cast<unsigned long long>((keys[i] >> begin_bit) & mask)
                       << kSmallPositionBits) |
                        i
                    : ~0ull;
  __syncthreads();
  for (unsigned size = 2; size <= m; size *= 2) {
    for (unsigned d = size / 2; d > 0; d /= 2) {
      unsigned const t = threadIdx.x;
      if (t < m / 2) {
        unsigned const i = 2 * t - (t & (d - 1)), j = i + d;
        unsigned long long const a = word[i], b = word[j];
        if ((a > b) == ((i & size) == 0)) {
          word[i] = b;
          word[j] = a;
        }
      }
      __syncthreads();
    }
  }
  K k[2];
  uint32_t v[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    unsigned const i = threadIdx.x + r * kSmallBlock;
    if (i < n) {
      unsigned const p = static_cast<unsigned>(word[i]) & (kSmallSort - 1u);
      k[r]             = keys[p];
      v[r]             = iota_vals ? p + iota_base : vals[p];
    }
  }
  __syncthreads();  // the pairs are read before they are overwritten
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    unsigned const i = threadIdx.x + r * kSmallBlock;
    if (i < n) {
      keys[i] = k[r];
      vals[i] = v[r];
    }
  }
}

template <typename K>
bool radix_sort_pairs(K* keys, uint32_t* vals, K* keys_alt, uint32_t* vals_alt, size_t n,
                      int begin_bit, int end_bit, bool iota_vals, Allocator const& alloc,
                      uint32_t iota_base = 0)
{
  int const width = end_bit - begin_bit;
  if (n > 0 && n <= kSmallSort && width > 0 && width <= 64 - kSmallPositionBits) {
    K const mask = width >= static_cast<int>(8 * sizeof(K)) ? static_cast<K>(~K{0})
                                                             : static_cast<K>((K{1} << width) - 1u);
    small_sort_kernel<K><<<1, kSmallBlock, 0, alloc.stream()>>>(
      keys, vals, static_cast<unsigned>(n), begin_bit, mask, iota_vals, iota_base);
    CSPT_CHECK_LAUNCH();
    return false;
  }
  unsigned const ntiles = static_cast<unsigned>((n + kSortTile - 1) / kSortTile);
  return radix_sort_tiles<K>(keys, vals, keys_alt, vals_alt, n, begin_bit, end_bit, iota_vals,
                             PlainTiles{n, ntiles}, ntiles, alloc, iota_base);
}

// The same within segments: tiles (device) never cross a segment boundary
// and cover [0, n); each segment is sorted in place by bits [begin_bit,
// end_bit).
template <typename K>
bool radix_sort_segments(K* keys, uint32_t* vals, K* keys_alt, uint32_t* vals_alt, size_t n,
                         int begin_bit, int end_bit, bool iota_vals, SortTile const* tiles,
                         unsigned ntiles, Allocator const& alloc)
{
  return radix_sort_tiles<K>(keys, vals, keys_alt, vals_alt, n, begin_bit, end_bit, iota_vals,
                             SegmentTiles{tiles}, ntiles, alloc);
}

// Tiles of at most kSortTile items over segments [bounds[j], bounds[j+1])
// (host; empty segments get none).
inline void segment_sort_tiles(std::vector<uint64_t> const& bounds, std::vector<SortTile>& out)
{
  out.clear();
  for (size_t j = 0; j + 1 < bounds.size(); ++j) {
    uint64_t const b = bounds[j], e = bounds[j + 1];
    if (e <= b) continue;
    uint32_t const first = static_cast<uint32_t>(out.size());
    uint32_t const count = static_cast<uint32_t>((e - b + kSortTile - 1) / kSortTile);
    for (uint32_t k = 0; k < count; ++k) {
      uint64_t const tb = b + static_cast<uint64_t>(k) * kSortTile;
      uint64_t const te = tb + kSortTile < e ? tb + kSortTile : e;
      out.push_back(SortTile{static_cast<uint32_t>(tb), static_cast<uint32_t>(te), first, count});
    }
  }
}

// ---------------------------------------------------------------------------
// Stable merge of sorted runs (merge path), for data sorted chunk by chunk as
// it arrives.  A pass merges runs 2k and 2k+1 of `src` into `dst` (an
// unpaired last run is copied).  Each block owns kMergeTile outputs of one
// pair: it finds where its diagonal range starts and ends in the two runs
// (ties go to the left run, whose positions come first), stages both slices
// in shared memory, merges kMergeItems outputs per thread and writes the tile
// out in order.
// ---------------------------------------------------------------------------
constexpr int kMergeBlock   = 256;
constexpr int kMergeItems   = 8;
constexpr int kMergeTile    = kMergeBlock * kMergeItems;
constexpr int kMaxMergePairs = 8;

struct MergePair {
  uint32_t a0, na, nb;  // left run [a0, a0 + na), right run [a0 + na, a0 + na + nb)
  uint32_t tile0;       // the pair's first output tile
};
struct MergePlan {
  MergePair p[kMaxMergePairs];
  int n;
};

// outputs taken from a among the first d of the stable merge of a and b
template <typename K>
__device__ inline uint32_t merge_split(K const* a, uint32_t na, K const* b, uint32_t nb,
                                       uint32_t d)
{
  uint32_t lo = d > nb ? d - nb : 0u, hi = d < na ? d : na;
  while (lo < hi) {
    uint32_t const mid = (lo + hi) >> 1;
    if (a[mid] <= b[d - 1 - mid])
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

template <typename K>
__global__ void __launch_bounds__(kMergeBlock)
  merge_runs_kernel(K const* __restrict__ ks, uint32_t const* __restrict__ vs, K* __restrict__ kd,
                    uint32_t* __restrict__ vd, MergePlan plan)
{
  __shared__ K sk[kMergeTile];
  __shared__ uint32_t sv[kMergeTile];
  __shared__ uint32_t split[2];
  int p = 0;
  while (p + 1 < plan.n && plan.p[p + 1].tile0 <= blockIdx.x) ++p;
  MergePair const P = plan.p[p];
  uint32_t const n  = P.na + P.nb;
  uint32_t const d0 = (blockIdx.x - P.tile0) * static_cast<uint32_t>(kMergeTile);
  uint32_t const d1 = min(n, d0 + static_cast<uint32_t>(kMergeTile));
  K const* a        = ks + P.a0;
  K const* b        = a + P.na;
  if (threadIdx.x == 0) split[0] = merge_split(a, P.na, b, P.nb, d0);
  if (threadIdx.x == 32) split[1] = merge_split(a, P.na, b, P.nb, d1);
  __syncthreads();
  uint32_t const i0 = split[0], i1 = split[1];
  uint32_t const la = i1 - i0, lb = (d1 - i1) - (d0 - i0);
  uint32_t const j0 = d0 - i0;
  for (uint32_t t = threadIdx.x; t < la; t += kMergeBlock) {
    sk[t] = a[i0 + t];
    sv[t] = vs[P.a0 + i0 + t];
  }
  for (uint32_t t = threadIdx.x; t < lb; t += kMergeBlock) {
    sk[la + t] = b[j0 + t];
    sv[la + t] = vs[P.a0 + P.na + j0 + t];
  }
  __syncthreads();
  uint32_t const m  = d1 - d0;
  uint32_t const ld = threadIdx.x * kMergeItems;
  K okey[kMergeItems];
  uint32_t oval[kMergeItems];
  if (ld < m) {
    uint32_t i = merge_split(sk, la, sk + la, lb, ld), j = ld - i;
#pragma unroll
    for (int k = 0; k < kMergeItems; ++k) {
      if (ld + k < m) {
        bool const left = j >= lb || (i < la && sk[i] <= sk[la + j]);
        okey[k]         = left ? sk[i] : sk[la + j];
        oval[k]         = left ? sv[i] : sv[la + j];
        i += left ? 1u : 0u;
        j += left ? 0u : 1u;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kMergeItems; ++k) {
    if (ld + k < m) {
      sk[ld + k] = okey[k];
      sv[ld + k] = oval[k];
    }
  }
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < m; t += kMergeBlock) {
    kd[P.a0 + d0 + t] = sk[t];
    vd[P.a0 + d0 + t] = sv[t];
  }
}

// Merges the sorted runs [bounds[r], bounds[r+1]) of (keys, vals) into one
// (at most 2 kMaxMergePairs runs); returns true when the result is in the
// _alt buffers.
template <typename K>
bool merge_sorted_runs(K* keys, uint32_t* vals, K* keys_alt, uint32_t* vals_alt,
                       std::vector<size_t> bounds, cudaStream_t s)
{
  CSPT_EXPECTS(bounds.size() >= 2 && bounds.size() - 1 <= 2 * kMaxMergePairs,
               "too many sorted runs to merge");
  bool in_alt = false;
  while (bounds.size() > 2) {
    K const* ks        = in_alt ? keys_alt : keys;
    uint32_t const* vs = in_alt ? vals_alt : vals;
    K* kd              = in_alt ? keys : keys_alt;
    uint32_t* vd       = in_alt ? vals : vals_alt;
    size_t const runs  = bounds.size() - 1;
    MergePlan plan{};
    std::vector<size_t> next{bounds[0]};
    uint32_t tiles = 0;
    size_t r       = 0;
    for (; r + 1 < runs; r += 2) {
      uint32_t const na = static_cast<uint32_t>(bounds[r + 1] - bounds[r]);
      uint32_t const nb = static_cast<uint32_t>(bounds[r + 2] - bounds[r + 1]);
      plan.p[plan.n++]  = MergePair{static_cast<uint32_t>(bounds[r]), na, nb, tiles};
      tiles += (na + nb + kMergeTile - 1) / kMergeTile;
      next.push_back(bounds[r + 2]);
    }
    if (r < runs) {  // the unpaired last run
      size_t const b0 = bounds[r], m = bounds[r + 1] - bounds[r];
      CSPT_CUDA_TRY(cudaMemcpyAsync(kd + b0, ks + b0, m * sizeof(K), cudaMemcpyDeviceToDevice, s));
      CSPT_CUDA_TRY(
        cudaMemcpyAsync(vd + b0, vs + b0, m * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
      next.push_back(bounds[r + 1]);
    }
    if (tiles) {
      merge_runs_kernel<K><<<tiles, kMergeBlock, 0, s>>>(ks, vs, kd, vd, plan);
      CSPT_CHECK_LAUNCH();
    }
    bounds = std::move(next);
    in_alt = !in_alt;
  }
  return in_alt;
}

}  // namespace cspt
