// Small blocks cut from slabs of an upstream allocator.  Plain C++, so that the
// host tests can check it.
//
// Blocks are reused by size: powers of two, or, `fine`, multiples of 256 bytes at
// most a quarter larger than asked for (what is kept wastes less, what is short-lived
// is reused less).  Slabs double from first_slab to kLastSlab; there are at most
// kMaxSlabs, `most` bytes in all.  take() returns null where a block is beyond
// kMaxBlock or there is no memory for a slab: the caller then asks the upstream
// itself.  give() allocates nothing: take() has made room for
// every block it ever handed out.
#pragma once

#include <cstddef>
#include <vector>

namespace cspt {

// Upstream: void* allocate(size_t) (null where it has none), deallocate(void*, size_t).
template <typename Upstream>
class SlabArena {
 public:
  static constexpr size_t kMinBlock = 256, kMaxBlock = size_t{4} << 20;
  static constexpr size_t kLastSlab = size_t{32} << 20;
  static constexpr int kMaxSlabs = 8;

  SlabArena(Upstream up, size_t first_slab, size_t most, bool fine)
    : up_(up), first_slab_(first_slab), next_slab_(first_slab), most_(most), fine_(fine)
  {
  }
  ~SlabArena()
  {
    for (int i = 0; i < nslabs_; ++i) up_.deallocate(slabs_[i].p, slabs_[i].bytes);
  }
  SlabArena(SlabArena const&)            = delete;
  SlabArena& operator=(SlabArena const&) = delete;

  void* take(size_t bytes)
  {
    if (bytes > kMaxBlock) return nullptr;
    size_t size;
    Class& k = classes_[size_class(bytes, size)];
    if (k.free.empty()) {
      if (k.made == k.free.capacity()) k.free.reserve(2 * k.made + 8);
      if (static_cast<size_t>(end_ - at_) < size && !grow(size)) return nullptr;
      char* const p = at_;
      at_ += size;
      ++k.made;
      ++slabs_[nslabs_ - 1].live;
      return p;
    }
    char* const p = k.free.back();
    k.free.pop_back();
    ++slab_of(p)->live;
    return p;
  }
  // false: not one of this arena's blocks
  bool give(void* p, size_t bytes)
  {
    Slab* const s = slab_of(p);
    if (!s) return false;
    --s->live;
    size_t size;
    classes_[size_class(bytes, size)].free.push_back(static_cast<char*>(p));
    return true;
  }
  bool owns(void const* p) const { return const_cast<SlabArena*>(this)->slab_of(p) != nullptr; }
  // Gives back the slabs that hold no block in use.
  void trim()
  {
    for (int i = nslabs_ - 1; i >= 0; --i) {
      Slab const s = slabs_[i];
      if (s.live != 0) continue;
      for (Class& k : classes_) {
        size_t kept = 0;
        for (char* const p : k.free)
          if (!s.holds(p)) k.free[kept++] = p;
        k.made -= k.free.size() - kept;
        k.free.resize(kept);
      }
      if (end_ == s.p + s.bytes) at_ = end_ = nullptr;
      for (int j = i; j + 1 < nslabs_; ++j) slabs_[j] = slabs_[j + 1];
      --nslabs_;
      up_.deallocate(s.p, s.bytes);
    }
    if (nslabs_ == 0) next_slab_ = first_slab_;
  }
  size_t slab_bytes() const
  {
    size_t n = 0;
    for (int i = 0; i < nslabs_; ++i) n += slabs_[i].bytes;
    return n;
  }

 private:
  struct Slab {
    char* p;
    size_t bytes;
    size_t live;  // blocks in use
    bool holds(void const* q) const
    {
      char const* const c = static_cast<char const*>(q);
      return c >= p && c < p + bytes;
    }
  };
  struct Class {
    std::vector<char*> free;
    size_t made = 0;  // blocks handed out or free
  };
  // 1, 2, 3 and 4 units of kMinBlock, then four sizes an octave
  static constexpr int kClasses = 52;
  static_assert(kMinBlock << 14 == kMaxBlock && kLastSlab >= kMaxBlock, "sizes");
  int size_class(size_t bytes, size_t& size) const
  {
    size_t const units = (bytes + kMinBlock - 1) / kMinBlock;
    int octave         = 2;  // 2^octave < units <= 2^(octave + 1)
    while ((size_t{2} << octave) < units) ++octave;
    if (!fine_) {
      size = kMinBlock;
      while (size < bytes) size *= 2;
      if (units > 4) return 4 * octave - 1;
      return units == 3 ? 3 : static_cast<int>(units) - 1;
    }
    size_t const step = units <= 4 ? 1 : size_t{1} << (octave - 2);
    size_t const k    = (units + step - 1) / step;  // 5 to 8 beyond 4 units
    size              = k * step * kMinBlock;
    return static_cast<int>(units <= 4 ? units - 1 : 4 * (octave - 1) + k - 5);
  }
  Slab* slab_of(void const* p)
  {
    for (int i = 0; i < nslabs_; ++i)
      if (slabs_[i].holds(p)) return &slabs_[i];
    return nullptr;
  }
  bool grow(size_t least)
  {
    if (nslabs_ == kMaxSlabs) return false;
    size_t const size = next_slab_ < least ? least : next_slab_;
    if (slab_bytes() + size > most_) return false;
    void* const p     = up_.allocate(size);
    if (!p) return false;
    next_slab_ = size < kLastSlab / 2 ? 2 * size : kLastSlab;
    slabs_[nslabs_++] = Slab{static_cast<char*>(p), size, 0};
    at_               = static_cast<char*>(p);
    end_              = at_ + size;
    return true;
  }

  Upstream up_;
  size_t first_slab_, next_slab_, most_;
  bool fine_;
  Slab slabs_[kMaxSlabs];
  int nslabs_ = 0;
  char *at_ = nullptr, *end_ = nullptr;  // the rest of the last slab
  Class classes_[kClasses];
};

}  // namespace cspt
